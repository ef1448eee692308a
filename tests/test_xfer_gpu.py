"""Fields go to the device and come back unchanged (FP32: rounded once), whatever
way they take: under and over the staged copies' smallest size, whole and broken
chunks and pieces, rows longer than a chunk, rows either side of the length that
goes straight into the padded field, caller rows with a gap (Qx and Qy), pinned
memory, and several threads at once."""
import threading

import numpy as np
import pytest

from adaptflood_b200 import scenarios as sc
from adaptflood_b200.batch import Batch
from adaptflood_b200.sim import Simulation

pytestmark = pytest.mark.gpu


def _round_trip(nx, ny, prec, seed, pin=False):
    rng = np.random.default_rng(seed)
    f = {"H": rng.random((ny, nx)), "Qx": rng.normal(size=(ny + 1, nx + 1)), "Qy": rng.normal(size=(ny + 1, nx + 1))}
    f["Qx"][-1], f["Qy"][:, -1] = 0.0, 0.0
    with Simulation(sc.Case(nx, ny, 5.0, np.zeros((ny, nx))), prec) as s:
        if pin:
            import torch
            f = {k: torch.from_numpy(v).pin_memory().numpy() for k, v in f.items()}
        s.set_state(f["H"], f["Qx"], f["Qy"], 0.0)
        got = s.state()
    for k, v in f.items():
        np.testing.assert_array_equal(got[k], v if prec == "f64" else v.astype(np.float32).astype(np.float64))


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("nx,ny", [(7, 5), (511, 512), (513, 520), (1000, 1100), (2047, 700), (2049, 1031),
                                   (32768, 33), (140001, 9), (131072, 17), (524300, 3), (70001, 31), (37, 20000)])
def test_round_trip(cuda, prec, nx, ny):
    _round_trip(nx, ny, prec, nx + ny)


def test_round_trip_from_pinned_memory(cuda):
    _round_trip(1201, 907, "f64", 1, pin=True)


def test_round_trips_from_several_threads(cuda):
    bad = []

    def go(k):
        try:
            for r in range(3):
                _round_trip(900 + 31 * k, 700 + 17 * r, "f32" if k % 2 else "f64", 10 * k + r)
        except BaseException as e:  # noqa: BLE001
            bad.append(e)

    th = [threading.Thread(target=go, args=(k,)) for k in range(4)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not bad, bad


def test_rows_longer_than_the_staging_buffer(cuda):
    nx, ny = (64 << 20) // 8 + 1001, 2
    h = np.random.default_rng(5).random((ny, nx)).astype(np.float32).astype(np.float64)
    with Batch("f32", arena_bytes=2 << 30) as b:
        k = b.add(sc.Case(nx, ny, 5.0, np.full((ny, nx), -50.0), h0=h, sim_time=0.0))
        b.run()
        np.testing.assert_array_equal(b.depth(k), h)
    _round_trip(nx, ny, "f32", 5)


def test_batch_members_round_trip(cuda):
    rng = np.random.default_rng(3)
    cases = []
    for nx, ny in ((300, 200), (1025, 600), (64, 5000)):
        c = sc.Case(nx, ny, 5.0, np.full((ny, nx), -50.0), h0=rng.random((ny, nx)), sim_time=0.0)
        cases.append(c)
    with Batch("f64", arena_bytes=1 << 30) as b:
        slots = [b.add(c) for c in cases]
        b.run()
        for c, k in zip(cases, slots):
            np.testing.assert_array_equal(b.depth(k), c.h0)
