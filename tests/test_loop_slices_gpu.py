"""A call's steps in several launches of a whole-loop kernel: long calls give the
step kernel's results bit for bit (state, clock, step count, report times; volumes
summed in another order to 1e-12), step limits are exact past the first launch,
and other work gets the GPU while a call runs: a second simulation's steps and
another stream's kernels are over long before it."""
import threading

import numpy as np
import pytest

from adaptflood_b200 import forcing as fc
from adaptflood_b200 import scenarios as sc
from adaptflood_b200.sim import Simulation

pytestmark = pytest.mark.gpu

MODES = pytest.mark.parametrize("mode", ["resident", "stream"])


def _sim(monkeypatch, mode, case, prec):
    monkeypatch.setenv("AF_SIM_LOOP", mode)
    s = Simulation(case, prec, forcing=fc.pack(case))
    monkeypatch.delenv("AF_SIM_LOOP")
    return s


def _film(nx, ny, seed=1):
    """Rain-fed sheet flow that stays wet however long it runs."""
    r = np.random.default_rng(seed)
    dem = 0.02 * (ny - 1 - np.arange(ny, dtype=np.float64))[:, None] + 0.01 * r.random((ny, nx))
    return sc.Case(nx, ny, 5.0, dem, h0=np.full((ny, nx), 0.03), sim_time=1e12, mass_int=50.0, south_free=True,
                   rain_times=np.array([0.0, 1e9]), rain_rates=np.array([5e-6, 5e-6]))


@MODES
@pytest.mark.parametrize("prec", ["f64", "f32"])
def test_long_calls_equal_the_step_kernel(cuda, monkeypatch, mode, prec):
    case = sc.small_case(70, 40, seed=9, sim_time=600.0, channel=False, rain=True, n_qvar=2, n_hvar=1, n_qfix=2)
    case.mass_int = 90.0
    with _sim(monkeypatch, mode, case, prec) as a, _sim(monkeypatch, "graph", case, prec) as b:
        for t_stop, most in ((1e12, 4001), (1e12, 1999), (a.t + 9000.0, 1 << 40), (1e12, 1)):
            assert a.run(t_stop, most) == b.run(t_stop, most)
            assert a.status() == b.status()
        x, y = a.state(), b.state()
        for k in ("H", "Qx", "Qy"):
            np.testing.assert_array_equal(x[k], y[k], err_msg=k)
        ma, mb = a.mass_series(), b.mass_series()
        np.testing.assert_array_equal(ma[0], mb[0])
        np.testing.assert_allclose(ma[1:], mb[1:], rtol=1e-12, atol=0.0)


@MODES
def test_other_work_runs_beside_a_long_call(cuda, monkeypatch, mode):
    import torch
    with _sim(monkeypatch, mode, _film(700, 600), "f32") as a, _sim(monkeypatch, mode, _film(90, 80), "f32") as b:
        x = torch.zeros(1 << 20, device="cuda")
        x += 1.0  # a kernel's first launch loads it, which may wait for all that runs
        a.run(1e12, 10)
        a.launch(1e12, 200_000)  # more than a second
        running = torch.cuda.ExternalStream(a.stream)
        assert b.run(1e12, 50) == 50
        assert not running.query()
        for _ in range(5):
            x += 1.0
        torch.cuda.current_stream().synchronize()
        assert not running.query()
        a.sync()
        assert a.steps == 200_010 and float(x[0]) == 6.0


@MODES
def test_other_work_runs_beside_a_call_that_waits(cuda, monkeypatch, mode):
    with _sim(monkeypatch, mode, _film(700, 600), "f32") as a, _sim(monkeypatch, mode, _film(90, 80), "f32") as b:
        a.run(1e12, 10)
        long = threading.Thread(target=a.run, args=(1e12, 100_000))
        long.start()
        for _ in range(20):
            assert b.run(1e12, 50) == 50
        assert long.is_alive()
        long.join()
        assert a.steps == 100_010


@MODES
def test_calls_of_one_to_many_launches_end_where_they_should(cuda, monkeypatch, mode):
    """Step limits and stop times around the launches of a call, waiting or not."""
    case = _film(64, 50)
    with _sim(monkeypatch, mode, case, "f64") as a, _sim(monkeypatch, mode, case, "f64") as b:
        dt = 0.0
        for steps in (1, 700, 3000, 9000, 30_000):
            n0 = a.steps
            assert a.run(1e12, steps) == steps
            b.launch(1e12, steps)
            b.sync()
            assert a.status() == b.status() and a.steps == n0 + steps
            dt = a.status()[1]
            stop = a.t + 0.37 * steps * dt
            n = a.run(stop)
            b.launch(stop)
            b.sync()
            assert a.status() == b.status() and a.t >= stop and 0 < n < steps + 2
            assert a.t - a.status()[1] < stop  # no step past the one that reached it
        np.testing.assert_array_equal(a.depth(), b.depth())


def test_two_simulations_in_two_threads(cuda, monkeypatch):
    """Each gets the results it gets alone."""
    cases = [(_film(500, 300, 2), "f32", 6000), (_film(310, 290, 3), "f64", 3000)]
    alone = []
    for c, prec, steps in cases:
        with Simulation(c, prec) as s:
            s.run(1e12, steps)
            alone.append((s.status(), s.depth()))
    got = [None, None]

    def work(k):
        c, prec, steps = cases[k]
        with Simulation(c, prec) as s:
            s.run(1e12, steps)
            got[k] = (s.status(), s.depth())

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for (sa, ha), (sb, hb) in zip(alone, got):
        assert sa == sb
        np.testing.assert_array_equal(ha, hb)
