"""What the resident loop's warps read between a step's two barriers does not
depend on when they read it.  In a test build (build.build_late_test) all warps
but the block's first, which meanwhile sets the next step's time and dt, come 20
us late: the hydrographs, stage boundaries and rain must still be those of the
step's own time, so the state is the step kernel's bit for bit."""
import os
import subprocess
import sys
import textwrap

import pytest

from adaptflood_b200 import build as B

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = textwrap.dedent("""
    import os
    import sys
    sys.path.insert(0, {root!r})
    import numpy as np
    from adaptflood_b200 import _lib, forcing as fc, scenarios as sc
    from adaptflood_b200.sim import Simulation
    assert _lib.LIB_PATH.endswith("libadaptflood_latetest.so"), _lib.LIB_PATH
    case = sc.small_case(97, 300, seed=3, sim_time=80.0, rain=True, n_qvar=6, n_hvar=2, n_qfix=2)
    f = fc.pack(case)
    for prec in ("f64", "f32"):
        got = []
        for mode in ("resident", "graph"):
            os.environ["AF_SIM_LOOP"] = mode
            with Simulation(case, prec, forcing=f) as s:
                s.run(case.sim_time)
                got.append((s.status(), s.state()))
        assert got[0][0] == got[1][0], got
        for k in ("H", "Qx", "Qy"):
            np.testing.assert_array_equal(got[0][1][k], got[1][1][k], err_msg=prec + " " + k)
    print("same")
""")


def test_late_warps_look_up_the_same_time(cuda):
    B.build_late_test()  # incremental
    env = dict(os.environ, AF_LIB_PATH=B.LATETEST_LIB)
    r = subprocess.run([sys.executable, "-c", CHILD.format(root=ROOT)], env=env, capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.split() == ["same"], r.stderr[-3000:]
