"""Faces whose old discharges are not finite give the reference's values in every
FP64 kernel: infinities of either sign alone and as opposite pairs in a face's
transverse average (whose sum is a NaN with its sign bit set), NaNs of either
sign, and a NaN depth.  One step from a given state against the C oracle; the
tolerance is the one of the finite faces (1e-15 of a discharge: the oracle's pow
differs from the kernels' by one ulp on some depths), NaNs and infinities must be
where the oracle has them.  The fused step leaves out the reference's 0 * (qup +
qdown) of theta = 1, which is NaN beside a face that is not finite; its interior
faces are compared with the same law written without that term."""
import numpy as np
import pytest

from adaptflood_b200 import forcing as fc
from adaptflood_b200 import kernels as K
from adaptflood_b200 import scenarios as sc
from adaptflood_b200.batch import Batch
from adaptflood_b200.sim import Simulation
from oracle import oracle as orc

pytestmark = pytest.mark.gpu

NX, NY = 67, 40
NEG_NAN = np.copysign(np.nan, -1.0)


def _inputs(kind):
    rng = np.random.default_rng(5)
    c = sc.Case(NX, NY, 5.0, rng.uniform(0.0, 0.3, (NY, NX)), mass_int=0.0, east_free=True, south_free=True)
    h = rng.uniform(0.1, 0.5, (NY, NX))
    qx, qy = (rng.normal(0.0, 0.3, (NY + 1, NX + 1)) for _ in range(2))
    qx[-1, :] = 0.0
    qy[:, -1] = 0.0
    at = [(3, 4), (11, 31), (20, 33), (31, 62)]  # rows, columns: inside a strip and at its edges
    for j, i in at:
        if kind == "inf":
            qx[j, i], qy[j + 3, i] = np.inf, -np.inf
        elif kind == "pair":  # two of the four transverse discharges of a face
            qx[j, i], qx[j + 1, i] = np.inf, -np.inf
            qy[j + 4, i], qy[j + 4, i + 1] = -np.inf, np.inf
        elif kind == "nan":
            qx[j, i], qy[j + 3, i] = np.nan, NEG_NAN
        elif kind == "neg_nan":
            qx[j, i], qy[j + 3, i] = NEG_NAN, np.nan
        else:
            h[j, i] = np.nan
            h[j + 4, i] = NEG_NAN
    return c, h, qx, qy


def _law(c, dt, z0, h0, z1, h1, q0, a):
    """src/kernels.cpp:60-84 at theta = 1 without 0 * (qup + qdown); a = the four transverse discharges."""
    y0, y1 = z0 + h0, z1 + h1
    hf = np.where(y0 > y1, y0, y1) - np.where(z0 > z1, z0, z1)
    hf = np.where(hf > 0.0, hf, 0.0)
    hf = np.where(hf < 10.0, hf, 10.0)
    q0, a = q0 * (1.0 / c.dx), [k * (1.0 / c.dx) for k in a]
    av = (a[0] + a[1] + a[2] + a[3]) / 4.0
    gdt = 9.81 * dt
    with np.errstate(all="ignore"):
        num = (q0 + 0.0) - gdt * hf * (-(y0 - y1) / c.dx)
        den = 1.0 + gdt * hf * c.fpn * c.fpn * np.sqrt(q0 * q0 + av * av) / hf ** (10.0 / 3.0)
        return np.where(hf > c.depth_thresh, num / den * c.dx, 0.0)


def _fused(c, dt, h, qx, qy, want):
    """The oracle's discharges with the interior faces by _law."""
    z, X, Y = c.dem, qx[:NY], qy[:, :NX]
    out = {k: want[k].copy() for k in ("Qx", "Qy")}
    with np.errstate(all="ignore"):
        out["Qx"][:NY, 1:NX] = _law(c, dt, z[:, :-1], h[:, :-1], z[:, 1:], h[:, 1:], X[:, 1:-1],
                                    (Y[:-1, :-1], Y[:-1, 1:], Y[1:, :-1], Y[1:, 1:]))
        out["Qy"][1:NY, :NX] = _law(c, dt, z[:-1], h[:-1], z[1:], h[1:], Y[1:-1],
                                    (X[:-1, :-1], X[:-1, 1:], X[1:, :-1], X[1:, 1:]))
    return out


def _same(got, want, what):
    for k in ("Qx", "Qy"):
        np.testing.assert_allclose(got[k], want[k], rtol=1e-15, atol=0.0, err_msg=what + " " + k)


KINDS = pytest.mark.parametrize("kind", ["inf", "pair", "nan", "neg_nan", "nan_depth"])


@KINDS
@pytest.mark.parametrize("mode", ["resident", "stream", "graph"])
def test_one_step_from_a_state_that_is_not_finite(cuda, monkeypatch, mode, kind):
    c, h, qx, qy = _inputs(kind)
    f = fc.pack(c)
    o = orc.OracleSim(c, f)
    o.set_state(h, qx, qy, 0.0)
    o.run(1e30, 1)
    want = o.state(velocity=False)
    faces = _fused(c, o.t, h, qx, qy, want)
    lost = {k: np.isnan(want[k]) & ~np.isnan(faces[k]) for k in faces}
    for k in faces:  # the law is the oracle's, but for the term left out
        np.testing.assert_allclose(faces[k][~lost[k]], want[k][~lost[k]], rtol=1e-15, atol=0.0)
        assert np.isnan(faces[k]).any()
    nan = {k: np.isnan(v) for k, v in faces.items()}
    wet = nan["Qx"][:NY, :-1] | nan["Qx"][:NY, 1:] | nan["Qy"][:-1, :NX] | nan["Qy"][1:, :NX] | np.isnan(h)
    monkeypatch.setenv("AF_SIM_LOOP", mode)
    with Simulation(c, "f64", forcing=f) as s:
        s.set_state(h, qx, qy, 0.0)
        s.run(1e30, 1)
        got = s.state()
        assert s.status()[1] == o.t
    _same(got, faces, mode)
    np.testing.assert_array_equal(np.isnan(got["H"]), wet)


@KINDS
def test_dropin_faces_from_a_state_that_is_not_finite(cuda, kind):
    import torch
    c, h, qx, qy = _inputs(kind)
    f = fc.pack(c)
    o = orc.OracleSim(c, f)
    o.set_state(h, qx, qy, 0.0)
    o.run(1e30, 1)
    want = o.state(velocity=False)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a).reshape(-1)).cuda()  # noqa: E731
    H, Z, X, Y = dev(h), dev(c.dem), dev(qx), dev(qy)
    Xo, Yo = torch.zeros_like(X), torch.zeros_like(Y)
    K.UpdateQs_GPU(X, Y, Xo, Yo, NX, NY, c.dx)
    dt = K.FloodplainQ_GPU(H, Z, X, Y, Xo, Yo, NX, NY, c.dx, c.dx, c.fpn, c.depth_thresh, 10.0, 1e-4, 0.0,
                           1.0, c.dx * c.dx, c.cfl, 9.81, c.init_tstep, 1.0, c.nodata)
    assert dt == o.t
    for q, k, inner in ((X, "Qx", np.s_[:NY, 1:NX]), (Y, "Qy", np.s_[1:NY, :NX])):
        np.testing.assert_allclose(q.cpu().numpy().reshape(NY + 1, NX + 1)[inner], want[k][inner], rtol=1e-15,
                                   atol=0.0, err_msg=k)


def test_batch_member_with_a_depth_that_is_not_finite(cuda):
    """A batch takes no discharges: a NaN depth reaches its faces and their neighbours."""
    c, h, _, _ = _inputs("nan_depth")
    c.h0 = h
    f = fc.pack(c)
    o = orc.OracleSim(c, f)
    o.run(1e30, 2)
    want = o.state(velocity=False)
    with Batch("f64", arena_bytes=1 << 28) as b:
        k = b.add(c, f)
        b.run(max_steps=2)
        got = b.state(k)
    _same(got, want, "batch")
    np.testing.assert_array_equal(np.isnan(got["H"]), np.isnan(want["H"]))
