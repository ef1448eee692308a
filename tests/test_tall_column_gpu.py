"""The tallest column that fits the grid of the drop-in flux kernels (65535 blocks of
8 rows of faces), against the C oracle; the face tolerance is the other drop-in
tests' (the oracle's pow is an ulp off on some depths: 1e-15 relative)."""
import ctypes as C

import numpy as np
import pytest

from adaptflood_b200 import kernels as K
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("theta", [1.0, 0.9])
@pytest.mark.parametrize("ny", [1, 2, 524280, 524281])
def test_one_column(cuda, ny, theta):
    import torch
    rng = np.random.default_rng(ny)
    H, Z = rng.uniform(0.0, 0.5, ny), rng.uniform(0.0, 0.3, ny)
    F = 2 * (ny + 1)
    q = [rng.normal(0.0, 0.3, F) for _ in range(2)]
    want = np.full(F, 7.0)
    lib = orc._oracle_lib()
    p = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731
    d = C.c_double
    lib.afo_qy.argtypes = [C.c_void_p] * 5 + [C.c_int] * 2 + [d] * 8
    lib.afo_find_hmax.argtypes = [C.c_void_p, C.c_void_p, C.c_long, d]
    lib.afo_timestep.argtypes = [d] * 6
    dt = lib.afo_timestep(lib.afo_find_hmax(p(H), p(Z), ny, -9999.0), 1e-3, 0.7, 5.0, 9.81, 3.0)
    lib.afo_qy(p(H), p(Z), p(want), p(q[0]), p(q[1]), 1, ny, 5.0, 0.05, 1e-3, 10.0, dt, 9.81, theta, -9999.0)
    dev = lambda a: torch.from_numpy(a).cuda()  # noqa: E731
    X, Y = dev(np.full(F, 7.0)), dev(np.full(F, 7.0))
    tg = K.FloodplainQ_GPU(dev(H), dev(Z), X, Y, dev(q[0]), dev(q[1]), 1, ny, 5.0, 5.0, 0.05, 1e-3, 10.0, 1e-4,
                           0.0, 1.0, 25.0, 0.7, 9.81, 3.0, theta, -9999.0)
    assert tg == dt
    np.testing.assert_allclose(Y.cpu().numpy(), want, rtol=1e-15, atol=0.0)
    assert bool((X == 7.0).all())
