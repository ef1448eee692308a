"""The one-pass face kernel of the drop-in FloodplainQ against the C oracle's two
loops: grids around its 32 x 8 blocks, one column, one row, theta other than 1
(the general kernels), a threshold that sends every face to the library forms,
nodata, and old discharges that are infinite beside a face (the reference's
0 * (qup + qdown) is then NaN).  The oracle's pow differs from the kernels' by one
ulp on about 1e-7 of depths, which moves a discharge by at most 1.2e-16 of itself:
1e-15 relative.  And dt, which the device works out, is the host's to the bit."""
import ctypes as C

import numpy as np
import pytest

from adaptflood_b200 import kernels as K
from oracle import oracle as orc

pytestmark = pytest.mark.gpu
ND = -9999.0


@pytest.mark.parametrize("nx,ny,theta,thresh,inf", [
    (1, 9, 1.0, 1e-3, False), (9, 1, 1.0, 1e-3, False), (31, 7, 1.0, 1e-3, False),
    (32, 8, 1.0, 1e-3, False), (33, 9, 1.0, 1e-3, True), (64, 65, 0.9, 1e-3, False),
    (70, 33, 1.0, 1e-12, False), (200, 131, 1.0, 1e-3, False), (40, 20, 1.0, 50.0, False)])
def test_faces_and_dt_match_the_oracle(cuda, nx, ny, theta, thresh, inf):
    import torch
    rng = np.random.default_rng(nx * 100 + ny)
    F = (nx + 1) * (ny + 1)
    H = rng.uniform(0.0, 0.5, nx * ny)
    H[rng.random(nx * ny) < 0.2] = 0.0
    Z = rng.uniform(0.0, 0.3, nx * ny)
    if nx * ny > 100:
        Z[rng.integers(0, nx * ny, 5)] = ND
    q = [rng.normal(0.0, 0.3, F) for _ in range(2)]
    if inf:
        q[0][5 + 3 * (nx + 1)] = np.inf
        q[1][12 + 4 * (nx + 1)] = -np.inf
    want = [np.full(F, 7.0), np.full(F, 7.0)]
    lib = orc._oracle_lib()
    p = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731
    d = C.c_double
    lib.afo_qx.argtypes = [C.c_void_p] * 5 + [C.c_int] * 2 + [d] * 8
    lib.afo_qy.argtypes = lib.afo_qx.argtypes
    lib.afo_find_hmax.argtypes = [C.c_void_p, C.c_void_p, C.c_long, d]
    lib.afo_timestep.argtypes = [d] * 6
    dt = lib.afo_timestep(lib.afo_find_hmax(p(H), p(Z), nx * ny, ND), thresh, 0.7, 5.0, 9.81, 3.0)
    for fn, w in ((lib.afo_qx, want[0]), (lib.afo_qy, want[1])):
        fn(p(H), p(Z), p(w), p(q[0]), p(q[1]), nx, ny, 5.0, 0.05, thresh, 10.0, dt, 9.81, theta, ND)
    dev = lambda a: torch.from_numpy(a).cuda()  # noqa: E731
    got = [dev(np.full(F, 7.0)), dev(np.full(F, 7.0))]
    tg = K.FloodplainQ_GPU(dev(H), dev(Z), got[0], got[1], dev(q[0]), dev(q[1]), nx, ny, 5.0, 5.0, 0.05,
                           thresh, 10.0, 1e-4, 0.0, 1.0, 25.0, 0.7, 9.81, 3.0, theta, ND)
    assert tg == dt
    for a, b in zip(got, want):
        np.testing.assert_allclose(a.cpu().numpy(), b, rtol=1e-15, atol=0.0)
