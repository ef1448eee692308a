"""What a simulation holds on the device: its field planes, its tables and its
loop's exchange, before and after fields went in and out; and where the device has
no room for the exchange, the simulation is made all the same and steps as any
other.  Fields that are read, or set to what they are, between steps change
nothing (transfers go through the planes that do not hold the state)."""
import ctypes as C

import numpy as np
import pytest

from adaptflood_b200 import forcing as fc
from adaptflood_b200 import scenarios as sc
from adaptflood_b200.sim import Simulation

pytestmark = pytest.mark.gpu


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def _pitch(nx, prec):
    n = 1 if prec == "f64" else 4
    return (-(-nx // (30 * n)) * 30 * n + n + 31) // 32 * 32


@pytest.mark.parametrize("prec,nx,ny", [("f32", 2500, 1801), ("f64", 1501, 1100), ("f32", 300, 200), ("f64", 2100, 900)])
def test_a_simulation_holds_its_planes_and_tables(cuda, prec, nx, ny):
    case = sc.Case(nx, ny, 5.0, np.zeros((ny, nx)), h0=np.full((ny, nx), 0.1))
    size = 8 if prec == "f64" else 4
    with Simulation(case, prec) as s:  # modules and pools that come with the first one
        s.run(1e12, 3)
    planes = 8 * (128 + (ny + 1) * _pitch(nx, prec)) * size
    # Special-cell offsets, partials, report series, exchange (its halo rows: [2][blocks][2][nx + 1] words of
    # 16 or 32 bytes on a grid that is held on chip) and the granularity of seven allocations.
    strips = -(-nx // (30 if prec == "f64" else 120)) * ny
    rest = 28 * strips + (2 << 20) + (1 << 20) + (4 * 148 * (nx + 1) * 4 * size if nx < 1000 else 0) + 7 * (2 << 20)
    before = _free()
    with Simulation(case, prec) as s:
        made = before - _free()
        assert made <= planes + rest, (made, planes, rest)
        s.set_state(np.full((ny, nx), 0.2), None, None, 0.0)
        s.run(1e12, 2)
        s.state()
        assert before - _free() <= made


@pytest.mark.parametrize("prec", ["f64", "f32"])
def test_made_without_room_for_the_exchange(cuda, prec):
    import torch
    nx, ny = 900, 148  # held on chip; its halo rows take 8.5 MB in FP32
    case = sc.small_case(nx, ny, seed=8, sim_time=60.0, rain=True)
    f = fc.pack(case)
    with Simulation(case, prec, forcing=f) as s:
        n = s.run(30.0)
        want = s.state()
    rt = C.CDLL("libcudart.so.12")
    hold = []

    def take(size):
        p = C.c_void_p()
        if rt.cudaMalloc(C.byref(p), C.c_size_t(size)) != 0:
            rt.cudaGetLastError()
            return False
        hold.append(p)
        return True

    planes = 8 * (128 + (ny + 1) * _pitch(nx, prec)) * (8 if prec == "f64" else 4)
    torch.cuda.empty_cache()
    try:
        for size in (1 << 30, 64 << 20, 2 << 20):
            while _free() - size > planes + (10 << 20) and take(size):
                pass
        with Simulation(case, prec, forcing=f) as s:
            assert s.run(30.0) == n
            got = s.state()
    finally:
        for p in hold:
            rt.cudaFree(p)
    for k in ("H", "Qx", "Qy"):
        np.testing.assert_array_equal(got[k], want[k])


@pytest.mark.parametrize("mode", ["resident", "stream", "graph"])
@pytest.mark.parametrize("prec,nx,ny", [("f32", 130, 61), ("f64", 95, 40), ("f64", 2049, 9), ("f32", 121, 33)])
def test_transfers_between_steps_change_nothing(cuda, monkeypatch, mode, prec, nx, ny):
    monkeypatch.setenv("AF_SIM_LOOP", mode)
    case = sc.small_case(nx, ny, seed=nx, sim_time=600.0, rain=True, nodata_block=True, h0=True, n_qvar=3,
                         n_hvar=1)
    f = fc.pack(case)
    with Simulation(case, prec, forcing=f) as a, Simulation(case, prec, forcing=f) as b:
        for k in range(7):
            a.run(1e12, 1)
            x = a.state()
            a.depth()
            if k % 3 == 2:
                a.set_state(x["H"], x["Qx"], x["Qy"], a.t)
        b.run(1e12, 7)
        assert a.status()[0] == b.status()[0]
        x, y = a.state(), b.state()
        for k in ("H", "Qx", "Qy"):
            np.testing.assert_array_equal(x[k], y[k], err_msg=k)
