"""The batch engine's own choice of strip heights and its per-step bookkeeping
(rain segments kept between steps, reports, finishing at different times) against
heights set by the caller and against each grid run alone: the same depths,
discharges, times and report times bit for bit, volumes (summed per strip) to
1e-12 relative."""
import numpy as np
import pytest

from adaptflood_b200 import scenarios as sc
from adaptflood_b200.batch import Batch
from adaptflood_b200.sim import Simulation

pytestmark = pytest.mark.gpu

# One strip or a few, one column of strips, many rounds of strips; the first
# of a size, one below and one above the lane widths.
SIZES = {"tiny": [(2, 2), (33, 7), (5, 200)], "mixed": [(121, 64), (700, 431), (64, 65), (3, 300), (317, 203)],
         "wide": [(2049, 700), (90, 90), (1500, 1101)]}


def _cases(sizes, knots):
    out = []
    for k, (nx, ny) in enumerate(sizes):
        rng = np.random.default_rng(100 * nx + ny)
        c = sc.Case(nx, ny, (2.0, 5.0, 10.0)[k % 3], rng.random((ny, nx)) * 2.0, h0=rng.random((ny, nx)),
                    sim_time=6.0 + 2.5 * k, mass_int=1.25)
        c.west_free = c.south_free = 1
        # Times that repeat (a step in the series), start late and end early; unsorted for some.
        t = np.sort(np.round(rng.uniform(0.5, 8.0, knots), 1))
        if k % 3 == 2:
            t = t[::-1].copy()
        c.rain_times, c.rain_rates = t, rng.random(knots) * 1e-5
        out.append(c)
    return out


@pytest.mark.parametrize("knots", [1, 2, 9])
@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("name", list(SIZES))
def test_members_do_not_depend_on_the_cut(cuda, name, prec, knots):
    cases = _cases(SIZES[name], knots)
    got = {}
    for how in ("auto", "fixed", "balanced"):
        with Batch(prec, arena_bytes=1 << 30) as b:
            if how == "fixed":
                b.set_balance(0)
            elif how == "balanced":
                b.set_balance(3)
            slots = [b.add(c) for c in cases]
            b.run()
            got[how] = [(b.state(s), b.status(s), b.mass_series(s)) for s in slots]
    alone = []
    for c in cases:
        with Simulation(c, prec) as s:
            s.run(c.sim_time)
            alone.append((s.state(), s.status(), s.mass_series()))
    for how, members in got.items():
        for (st, stat, m), (st1, stat1, m1) in zip(members, alone):
            for k in ("H", "Qx", "Qy"):
                np.testing.assert_array_equal(st[k], st1[k], err_msg=how + " " + k)
            assert tuple(stat)[:4] == tuple(stat1)[:4], how
            np.testing.assert_array_equal(m[0], m1[0])
            np.testing.assert_allclose(m[1], m1[1], rtol=1e-12)
            np.testing.assert_allclose(m[2], m1[2], rtol=1e-12)


def test_heights_set_by_the_caller_are_kept(cuda):
    c = _cases([(300, 200)], 2)[0]
    ref = None
    for rows in (None, 1, 7, 64):
        with Batch("f32", arena_bytes=1 << 28) as b:
            cls = int(np.log2(c.nx * c.ny))
            if rows:
                b.set_rows(cls, rows)
                assert b.rows(cls) == rows
            s = b.add(c)
            b.run()
            h = b.depth(s)
        ref = h if ref is None else ref
        np.testing.assert_array_equal(h, ref)
