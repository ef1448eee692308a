"""The straight-line FP64 face law and its hand-over to the library forms.

One step from a given state against the C oracle, at widths around a strip's 30
columns and with operands at and past the ends of the straight-line form's
range: a threshold below it (the whole step takes the library forms), tiny,
huge and zero discharges, depths past the clamp, flat water (exact zeros) and
equal cells whose quotients are exact.

The oracle takes the C library's pow, the kernels a restatement that differs
from it by one ulp on about 1e-7 of depths; one ulp there moves a discharge by
at most 1.2e-16 of itself through the denominator and its roundings, so each
face may differ by 1e-15 of its value, and a depth by that of the four fluxes'
volume or of itself.
"""
import numpy as np
import pytest

from adaptflood_b200 import forcing as fc
from adaptflood_b200 import scenarios as sc
from adaptflood_b200.sim import Simulation
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _state(nx, ny, kind, seed):
    rng = np.random.default_rng(seed)
    h = rng.uniform(0.0, 0.4, (ny, nx))
    h[rng.random((ny, nx)) < 0.2] = 0.0
    qx = rng.normal(0.0, 0.5, (ny + 1, nx + 1))
    qy = rng.normal(0.0, 0.5, (ny + 1, nx + 1))
    if kind == "tiny":
        qx *= 10.0 ** rng.uniform(-290, -100, qx.shape)
        qy *= 10.0 ** rng.uniform(-290, -100, qy.shape)
    elif kind == "huge":
        qx *= 10.0 ** rng.uniform(0, 45, qx.shape)
        qy *= 10.0 ** rng.uniform(0, 45, qy.shape)
    elif kind == "zero":
        qx[:] = 0.0
        qy[:] = 0.0
    elif kind == "deep":
        h += rng.uniform(5.0, 40.0, h.shape)
    qx[-1, :] = 0.0
    qy[:, -1] = 0.0
    return h, qx, qy


@pytest.mark.parametrize("nx,ny,kind,thresh,dx", [
    (2, 2, "plain", 1e-3, 10.0), (29, 5, "plain", 1e-3, 10.0), (30, 33, "plain", 1e-3, 2.0),
    (31, 32, "plain", 1e-3, 5.0), (60, 7, "zero", 1e-3, 3.0), (61, 65, "deep", 1e-3, 30.0),
    (91, 40, "tiny", 1e-3, 7.0), (90, 31, "huge", 1e-3, 10.0), (121, 9, "plain", 1e-12, 10.0),
    (45, 12, "tiny", 0.0, 0.1), (33, 20, "plain", 1e-3, 1e-12), (64, 64, "flat", 1e-3, 5.0)])
def test_one_step_matches_the_oracle(cuda, nx, ny, kind, thresh, dx):
    rng = np.random.default_rng(nx * 1000 + ny)
    dem = rng.uniform(0.0, 0.3, (ny, nx))
    if nx > 40:
        dem[ny // 2, nx // 3] = sc.NODATA
    c = sc.Case(nx, ny, dx, dem, depth_thresh=thresh, mass_int=0.0, east_free=True, south_free=True,
                west_free=nx % 2 == 0, north_free=nx % 3 == 0, rain_times=np.array([0.0, 1e6]),
                rain_rates=np.array([1e-5, 1e-5]))
    h, qx, qy = _state(nx, ny, kind, ny)
    if kind == "flat":
        c.dem[:] = 1.0
        h[:] = 0.25
        qx[:] = 0.0
        qy[:] = 0.0
    f = fc.pack(c)
    o = orc.OracleSim(c, f)
    o.set_state(h, qx, qy, 0.0)
    o.run(1e30, 1)
    want = o.state(velocity=False)
    with Simulation(c, "f64", forcing=f) as s:
        s.set_state(h, qx, qy, 0.0)
        s.run(1e30, 1)
        got = s.state()
        dt = s.status()[1]
    assert o.t == dt
    for k in ("Qx", "Qy"):
        np.testing.assert_allclose(got[k], want[k], rtol=1e-15, atol=0.0, err_msg=k)
    q = 4e-15 * dt / (dx * dx) * max(np.abs(want["Qx"]).max(), np.abs(want["Qy"]).max())
    np.testing.assert_allclose(got["H"], want["H"], rtol=1e-15, atol=q)
