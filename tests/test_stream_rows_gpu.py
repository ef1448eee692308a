"""The streamed loop's strip heights and its copy of the row loop without nodata
tests, against the graph of step kernels with bulk row copies: the same state bit
for bit and the same report times, volumes to 1e-12 relative (they are summed per
strip).  Heights: of the rule on either side of its limits, and forced ones with
short last strips; grids with and without nodata cells."""
import numpy as np
import pytest

from adaptflood_b200 import scenarios as sc
from adaptflood_b200.sim import Simulation

pytestmark = pytest.mark.gpu


def _run(case, prec, steps):
    with Simulation(case, prec) as s:
        s.run(1e30, steps)
        return s.state(), s.status(), s.mass_series()


@pytest.mark.parametrize("prec,nx,ny,rows", [("f32", 1025, 1024, None), ("f32", 2900, 2893, None), ("f32", 241, 9001, None),
                                             ("f32", 6001, 5600, None), ("f32", 1200, 901, 8), ("f32", 130, 77, 5),
                                             ("f64", 1201, 901, 8), ("f64", 4097, 4100, None)])
@pytest.mark.parametrize("holes", [False, True])
def test_streamed_loop_equals_step_kernels(cuda, monkeypatch, prec, nx, ny, rows, holes):
    rng = np.random.default_rng(nx + ny)
    z = rng.random((ny, nx))
    c = sc.Case(nx, ny, 5.0, z, h0=rng.random((ny, nx)), mass_int=0.5, west_free=True, north_free=True)
    if holes:
        z[ny // 3:ny // 3 + 3, :nx // 2] = c.nodata
        z[-1, -1] = z[0, 0] = c.nodata
    monkeypatch.setenv("AF_SIM_LOOP", "graph")
    monkeypatch.setenv("AF_SIM_TMA", "0")
    want, stat, mass = _run(c, prec, 7)
    monkeypatch.setenv("AF_SIM_LOOP", "stream")
    monkeypatch.delenv("AF_SIM_TMA")
    if rows:
        monkeypatch.setenv("AF_SIM_ROWS", str(rows))
    got, stat1, mass1 = _run(c, prec, 7)
    for k in ("H", "Qx", "Qy"):
        np.testing.assert_array_equal(got[k], want[k], err_msg=k)
    assert tuple(stat) == tuple(stat1)
    np.testing.assert_array_equal(mass1[0], mass[0])
    np.testing.assert_allclose(mass1[1], mass[1], rtol=1e-12)
    np.testing.assert_allclose(mass1[2], mass[2], rtol=1e-12)
