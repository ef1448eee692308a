"""A strip height set for a size class bounds the heights of the launches after it,
also where the members are already cut and taller strips are estimated faster: the
strips of each step, from the batch's own trace."""
import numpy as np
import pytest

from adaptflood_b200 import scenarios as sc
from adaptflood_b200.batch import Batch, size_class

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,cols", [("f32", 120), ("f64", 30)])
@pytest.mark.parametrize("rows", [3, 7, 20])
def test_a_height_set_between_launches_is_kept(cuda, prec, cols, rows):
    nx, ny = 1500, 1400
    c = sc.Case(nx, ny, 5.0, np.zeros((ny, nx)), h0=np.full((ny, nx), 0.1), sim_time=1e9)
    strips_x = -(-nx // cols)
    with Batch(prec, arena_bytes=1 << 30) as b:
        b.set_trace(64)
        b.add(c)
        b.run(max_steps=2)
        b.set_rows(size_class(nx, ny), rows)
        b.run(max_steps=2)
        units = [int(r[3]) for r in b.trace()]
    assert len(units) == 4
    assert all(u >= strips_x * -(-ny // rows) for u in units[2:]), units
