"""Fields on either side of the sizes that come back straight from the padded field
(FP64: at most 1 MB, and 128 rows or, of whole 32 bytes, 2048), whole and in the caller's gapped rows (Qx and Qy),
from simulations and batches: unchanged (FP32: rounded once)."""
import numpy as np
import pytest

from adaptflood_b200 import scenarios as sc
from adaptflood_b200.batch import Batch
from adaptflood_b200.sim import Simulation

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("nx,ny", [(2, 2), (20, 127), (20, 128), (20, 129), (1023, 127), (1023, 128), (1024, 128),
                                   (1025, 128), (1040, 126), (2047, 64), (2047, 65), (2048, 3),
                                   (20, 2047), (20, 2048), (20, 2049), (200, 655), (200, 656), (21, 128), (21, 129)])
def test_small_fields(cuda, prec, nx, ny):
    r = np.random.default_rng(nx + ny)
    f = {"H": r.random((ny, nx)), "Qx": r.normal(size=(ny + 1, nx + 1)), "Qy": r.normal(size=(ny + 1, nx + 1))}
    f["Qx"][-1], f["Qy"][:, -1] = 0.0, 0.0
    with Simulation(sc.Case(nx, ny, 5.0, np.zeros((ny, nx))), prec) as s:
        s.set_state(f["H"], f["Qx"], f["Qy"], 0.0)
        for _ in range(2):
            got = s.state()
            for k, v in f.items():
                np.testing.assert_array_equal(got[k], v if prec == "f64" else v.astype(np.float32).astype(np.float64))
    with Batch(prec, arena_bytes=1 << 28) as b:
        k = b.add(sc.Case(nx, ny, 5.0, np.full((ny, nx), -50.0), h0=f["H"], sim_time=0.0))
        b.run()
        h = f["H"] if prec == "f64" else f["H"].astype(np.float32).astype(np.float64)
        np.testing.assert_array_equal(b.depth(k), h)
