"""What a problem needs on the device, and what it does where there is no room for
more: the rest of the GPU is held by one allocation meanwhile."""
import gc

import numpy as np
import pytest

from felspa_b200 import abi, fields as F
from felspa_b200.level_set import AdvectSimulator, Mesh, Problem, ReinitSimulatorLDG
from felspa_b200.lib import FlspError, check, load

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

MB = 1 << 20


def free():
    gc.collect()   # problems that earlier tests left
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


class Rest:
    """holds all of the device's memory but `leave` bytes"""

    def __init__(self, leave):
        n = free() - int(leave)
        self.t = torch.empty(max(n, 1), dtype=torch.uint8, device="cuda:0")

    def give_back(self):
        self.t = None
        free()


def rate(sim):
    return sim.explicit_time_derivative(0.0)


def table_bytes(n, p):
    """a velocity table of a 3D FP32 problem: 4 x 4 x 4 tiles, 64 (p+2)^3 points of
    three components and 240 faces of (p+2)^2 points each"""
    tiles = np.prod([(v + 3) // 4 for v in n])
    return int(tiles) * 4 * (3 * 64 * (p + 2) ** 3 + 240 * (p + 2) ** 2)


def test_lattice_is_checked_without_a_second_one(flsp):
    n = (40, 40, 40)
    sim = AdvectSimulator(Mesh(3, n), 2, basis=abi.BASIS_Q, precision=abi.FP32)
    lattice = F.random_fe_lattice(n, 2, seed=1)
    had = free()
    sim.problem.set_velocity_fe(2, lattice)
    took = had - free()
    assert took <= table_bytes(n, 2) + lattice.nbytes + 8 * MB
    sim.problem.set_velocity_fe(2, -lattice)
    assert had - free() <= took + 2 * MB


def test_lattice_without_room_for_another(flsp):
    """degree 3 on degree-1 cells: the lattice is larger than the staging buffer,
    and there is room for one lattice and the table only"""
    n = (64, 64, 64)
    warm = AdvectSimulator(Mesh(3, (8, 8, 8)), 1, basis=abi.BASIS_P, precision=abi.FP32)
    warm.problem.project(F.sphere((0.5, 0.5, 0.5), 0.3))
    warm.problem.set_velocity_fe(3, F.random_fe_lattice((8, 8, 8), 3, seed=1))
    rate(warm)
    a, b = (F.random_fe_lattice(n, 3, seed=s) for s in (2, 3))
    sim = AdvectSimulator(Mesh(3, n), 1, basis=abi.BASIS_P, precision=abi.FP32)
    sim.problem.project(F.sphere((0.5, 0.5, 0.5), 0.3))
    assert a.nbytes > 100 * MB
    rest = Rest(a.nbytes + table_bytes(n, 1) + 60 * MB)
    try:
        sim.problem.set_velocity_fe(3, a)
        first = rate(sim)
        sim.problem.set_velocity_fe(3, b)
        second = rate(sim)
        bad = a.copy()
        bad.ravel()[-1] = np.inf
        with pytest.raises(FlspError, match="non-finite"):
            sim.problem.set_velocity_fe(3, bad)
        assert np.array_equal(rate(sim), second)
    finally:
        rest.give_back()
    for lattice, want in ((a, first), (b, second)):
        sim.problem.set_velocity_fe(3, lattice)
        assert np.array_equal(rate(sim), want)
    assert not np.array_equal(first, second)


def test_advection_without_room_for_the_sign_table(flsp):
    """P basis: the table of a reinitialisation (288 bytes a cell at 3D degree 2)
    is no condition for a problem that only advects"""
    n = (72, 72, 72)
    for warm in (True, False):
        if not warm:
            ndofs = 10 * int(np.prod(n))
            rest = Rest(ndofs * (3 * 4 + 6 * 8) + 60 * MB)
        try:
            pb = Problem(Mesh(3, (8, 8, 8) if warm else n), 2, basis=abi.BASIS_P, precision=abi.FP32, cfl_max=0.1)
            pb.set_velocity(F.deformation_3d())
            pb.project(F.sphere((0.4, 0.4, 0.4), 0.2))
            check(load().flsp_advance_steps(pb.h, 2, float("inf")))
            o = abi.default_reinit_opts(mode=abi.REINIT_FIXED, n_pseudo_steps=1)
            if warm:
                ReinitSimulatorLDG(pb).run_iteration(o)
                pb.close()
                continue
            before = pb.get_state()
            with pytest.raises(FlspError, match="sign table"):
                ReinitSimulatorLDG(pb).run_iteration(o)
            assert np.array_equal(pb.get_state(), before)
        finally:
            if not warm:
                rest.give_back()
    ReinitSimulatorLDG(pb).run_iteration(o)
    assert not np.array_equal(pb.get_state(), before)
    pb.close()
