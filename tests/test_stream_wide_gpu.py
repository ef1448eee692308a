"""Wide grids of fewer than 2^20 cells, which the streamed loop steps by default in
FP32 at the height of its rule: the same state as the graph of step kernels bit for
bit, with short last strips and short last columns of strips."""
import numpy as np
import pytest

from adaptflood_b200 import scenarios as sc
from adaptflood_b200.sim import Simulation

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(2000, 220), (4001, 199), (9000, 101), (1000, 1000), (30000, 32), (120001, 3)])
def test_wide_grids_equal_the_step_kernel(cuda, monkeypatch, nx, ny):
    r = np.random.default_rng(nx)
    c = sc.Case(nx, ny, 5.0, r.random((ny, nx)), h0=r.random((ny, nx)), mass_int=0.5, west_free=True, south_free=True)
    got = []
    for mode in ("", "graph"):
        if mode:
            monkeypatch.setenv("AF_SIM_LOOP", mode)
        with Simulation(c, "f32") as s:
            s.run(1e30, 7)
            got.append((s.status(), s.state()))
    assert got[0][0] == got[1][0]
    for k in ("H", "Qx", "Qy"):
        np.testing.assert_array_equal(got[0][1][k], got[1][1][k], err_msg=k)
