"""Special cells of the resident loop around what a block keeps of them in shared
memory (128 cells, 256 sources a band): at the limits and one past each, many sources in
one cell, with hydrographs and stage boundaries, against the step kernel bit for
bit.  On 148 rows a band is one row."""
import numpy as np
import pytest

from adaptflood_b200 import forcing as fc
from adaptflood_b200 import scenarios as sc
from adaptflood_b200.sim import Simulation

pytestmark = pytest.mark.gpu

NX, NY = 300, 148


def _points(row, cells, sources, seed):
    """`cells` special cells in a row; sources spread over them, the first with half of them."""
    r = np.random.default_rng(seed)
    cols = np.sort(r.choice(NX, cells, replace=False))
    out = []
    for k in range(sources):
        i = int(cols[0] if k < sources // 2 and sources > cells else cols[k % cells])
        if k % 3:
            tt, vv = sc.triangular_hydrograph(float(r.uniform(0.01, 0.1)), float(r.uniform(5, 20)), float(r.uniform(0, 10)))
            out.append(sc.PointBC(sc.QVAR, i, row, name="q%d_%d" % (row, k), times=tt, values=vv))
        else:
            out.append(sc.PointBC(sc.QFIX, i, row, value=float(r.uniform(-0.01, 0.1))))
    for k in range(0, cells, 7):
        tt = np.linspace(0.0, 60.0, 9)
        out.append(sc.PointBC(sc.HVAR, int(cols[k]), row, name="h%d_%d" % (row, k), times=tt,
                              values=0.3 + 0.2 * np.sin(tt / 5.0 + k)))
    return out


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("cells,sources", [(128, 128), (129, 129), (64, 256), (64, 257), (128, 256), (3, 600), (300, 300)])
def test_bands_with_many_special_cells(cuda, monkeypatch, prec, cells, sources):
    r = np.random.default_rng(cells + sources)
    case = sc.Case(NX, NY, 10.0, r.random((NY, NX)), sim_time=60.0, mass_int=9.0, south_free=True)
    for row in (0, 70, NY - 1):
        case.points += _points(row, cells, sources, row + cells)
    f = fc.pack(case)
    got = []
    for mode in ("resident", "graph"):
        monkeypatch.setenv("AF_SIM_LOOP", mode)
        with Simulation(case, prec, forcing=f) as s:
            s.run(1e12, 60)
            got.append((s.status(), s.state()))
    assert got[0][0] == got[1][0]
    for k in ("H", "Qx", "Qy"):
        np.testing.assert_array_equal(got[0][1][k], got[1][1][k], err_msg=k)
