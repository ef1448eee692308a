"""The time-out path of every loop, in the test build whose waits give up at once
(build.build_wait_test; see test_failure_gpu.py): the whole-loop launches with the
state on chip and in HBM (there a warp also drains its copies in mid-strip), the step
kernel's graph and the batch, in both precisions.  Each call ends with AF_ESTATE
after one step, the simulation stays stopped, and the process goes on using the
device."""
import os
import subprocess
import sys
import textwrap

import pytest

from adaptflood_b200 import _lib
from adaptflood_b200 import build as B

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = textwrap.dedent("""
    import ctypes as C
    import os
    import sys
    sys.path.insert(0, {root!r})
    import torch
    from adaptflood_b200 import _lib, forcing as fc, scenarios as sc
    from adaptflood_b200.batch import Batch
    from adaptflood_b200.sim import Simulation
    assert _lib.LIB_PATH.endswith("libadaptflood_waittest.so"), _lib.LIB_PATH
    case = sc.small_case(200, 150, seed=41, sim_time=200.0, rain=True)
    f = fc.pack(case)

    def code(fn):
        try:
            fn()
        except _lib.AFError as e:
            return e.code
        return 0

    for prec in ("f64", "f32"):
        for mode in ("resident", "stream", "graph"):
            os.environ["AF_SIM_LOOP"] = mode
            with Simulation(case, prec, forcing=f) as s:
                first = code(lambda: s.run(case.sim_time))
                steps = s.status()[3]
                print(prec, mode, first, steps, code(lambda: s.run(case.sim_time)), s.status()[3] - steps)
        with Batch(prec, arena_bytes=1 << 28) as b:
            b.add(case, f)
            print(prec, "batch", code(b.run))
        x = torch.zeros(1000, dtype=torch.float64, device="cuda")
        st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
        assert _lib.lib().af_fill(C.c_void_p(x.data_ptr()), 1000, 2.5, st) == 0
        assert float(x.sum()) == 2500.0
""")


def test_every_loop_times_out_with_estate(cuda):
    B.build_wait_test()  # incremental
    env = dict(os.environ, AF_LIB_PATH=B.WAITTEST_LIB)
    r = subprocess.run([sys.executable, "-c", CHILD.format(root=ROOT)], env=env, capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-3000:]
    e = _lib.AF_ESTATE
    want = []
    for prec in ("f64", "f32"):
        want += [f"{prec} {mode} {e} 1 {e} 0" for mode in ("resident", "stream", "graph")] + [f"{prec} batch {e}"]
    assert r.stdout.split("\n")[:-1] == want, r.stdout
