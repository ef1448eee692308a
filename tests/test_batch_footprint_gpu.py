"""A member's footprint in the batch's arena: no more per-strip words than one per
row and 16-byte-lane strip (60 columns in FP64, 120 in FP32), whatever the width of the
strips that step it, so that an arena holds the grids it always held; and the
lowest strips that leaves are used and give the results of any others."""
import numpy as np
import pytest

from adaptflood_b200 import scenarios as sc
from adaptflood_b200.batch import Batch, size_class

pytestmark = pytest.mark.gpu


def _footprint(nx, ny, prec):
    """Fields, tables of a case without points or rain, and per-strip words, each 256-byte aligned."""
    size, n = (8, 2) if prec == "f64" else (4, 4)
    strips_x = -(-nx // (30 * n))
    pitch = (strips_x * 30 * n + n + 31) // 32 * 32
    cells, qy = (128 + ny * pitch) * size, (128 + (ny + 1) * pitch) * size
    parts = [cells, cells, qy] * 2 + [cells] + [1] * 2 + [4] + [1] * 3 + [1] * 2 + [4] + [1] * 3 + [1] * 2
    parts += [4 * (strips_x * ny + 1), 1, 24 * strips_x * ny, 24 * 2]
    return sum(-(-p // 256) * 256 for p in parts)


@pytest.mark.parametrize("prec", ["f64", "f32"])
def test_footprint_is_bounded(cuda, prec):
    rng = np.random.default_rng(1)
    sizes = [(2, 2), (29, 3), (30, 2), (31, 2), (60, 5), (61, 7), (90, 4), (91, 101), (2048, 2048), (1501, 1101)]
    sizes += [(int(2 ** rng.uniform(1, 12)) + 2, int(2 ** rng.uniform(1, 12)) + 2) for _ in range(60)]
    with Batch(prec, arena_bytes=1 << 20) as b:
        for nx, ny in sizes:
            c = sc.Case(nx, ny, 5.0, np.zeros((ny, nx)), mass_int=0.0)
            assert b.footprint(c) <= _footprint(nx, ny, prec), (nx, ny)


def test_lowest_strips_give_the_same_results(cuda):
    ref = None
    for rows in (None, 1, 2, 5):
        with Batch("f64", arena_bytes=1 << 27) as b:
            got = []
            for nx, ny in ((61, 7), (91, 101), (120, 2), (29, 33)):
                c = sc.small_case(nx, ny, seed=nx, sim_time=20.0, rain=True, n_qvar=3, n_hvar=1)
                if rows:
                    b.set_balance(0)
                    b.set_rows(size_class(nx, ny), rows)
                got.append(b.add(c))
            b.run()
            got = [b.state(k) for k in got]
        ref = ref or got
        for x, y in zip(got, ref):
            for k in ("H", "Qx", "Qy"):
                np.testing.assert_array_equal(x[k], y[k])
