"""The loops in one launch -- small grids' state on chip, larger grids' in HBM --
give the step kernel's results bit for bit: fields, time, step counts and Hmax, at
bands of one and several rows, widths around a warp's 32 columns, more blocks
than rows and the other way round, run in pieces.  The volume reports add the
same depths in another order (FP64 sums of at most 2e5 terms: 1e-12 of the
volume)."""
import os

import numpy as np
import pytest

from adaptflood_b200 import forcing as fc
from adaptflood_b200 import scenarios as sc
from adaptflood_b200.sim import Simulation

pytestmark = pytest.mark.gpu

MODES = pytest.mark.parametrize("mode", ["resident", "stream"])


def _sim(monkeypatch, mode, case, prec, f):
    monkeypatch.setenv("AF_SIM_LOOP", mode)
    s = Simulation(case, prec, forcing=f)
    monkeypatch.delenv("AF_SIM_LOOP")
    return s


@MODES
@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("nx,ny,kw", [
    (2, 2, {}), (33, 3, dict(rain=True)), (31, 148, dict(free=(1, 0, 1, 0), n_hvar=1)),
    (64, 149, dict(rain=True, nodata_block=True)), (97, 300, dict(dup_sources=True, n_hfix=2, n_free_pts=1)),
    (500, 296, dict(rain=True, h0=True, n_qvar=5)), (32, 1000, dict(free=(0, 1, 0, 1), n_qfix=9)),
    (1200, 150, dict(free=(0, 0, 0, 0), h0=True, rain=True))])
def test_one_launch_loops_equal_the_step_kernel(cuda, monkeypatch, mode, prec, nx, ny, kw):
    case = sc.small_case(nx, ny, seed=nx + ny, sim_time=60.0, channel=False, **kw)
    case.mass_int = 7.0
    if nx == 500:
        case.h0 = sc.wet_start(case, channel_fill=0.3)
    f = fc.pack(case)
    with _sim(monkeypatch, mode, case, prec, f) as a, _sim(monkeypatch, "graph", case, prec, f) as b:
        for t_stop, most in ((60.0, 1), (60.0, 2), (60.0, 0), (25.0, 1 << 30), (20.0, 5), (60.0, 1 << 30)):
            assert a.run(t_stop, most) == b.run(t_stop, most)
            assert a.status() == b.status()
            x, y = a.state(), b.state()
            for k in ("H", "Qx", "Qy"):
                np.testing.assert_array_equal(x[k], y[k], err_msg=k)
        ta, va, aa = a.mass_series()
        tb, vb, ab = b.mass_series()
        np.testing.assert_array_equal(ta, tb)
        np.testing.assert_allclose(va, vb, rtol=1e-12, atol=0.0)
        np.testing.assert_allclose(aa, ab, rtol=1e-12, atol=0.0)


@MODES
def test_one_launch_loops_follow_set_state_and_restore(cuda, monkeypatch, tmp_path, mode):
    case = sc.small_case(120, 90, seed=4, sim_time=200.0, rain=True)
    f = fc.pack(case)
    path = os.path.join(tmp_path, "c.bin")
    with _sim(monkeypatch, mode, case, "f32", f) as a, _sim(monkeypatch, "graph", case, "f32", f) as b:
        a.run(100.0)
        a.checkpoint(path)
        a.run(200.0)
        b.restore(path)
        b.run(200.0)
        np.testing.assert_array_equal(a.depth(), b.depth())
        a.restore(path)
        a.run(200.0)
        np.testing.assert_array_equal(a.depth(), b.depth())
        for s in (a, b):
            s.set_state(np.full((90, 120), 0.1), None, None, 0.0)
            s.run(1e30, 7)
        np.testing.assert_array_equal(a.depth(), b.depth())
