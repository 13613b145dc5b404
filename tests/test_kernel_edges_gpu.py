"""The device kernels where a tile can go wrong: meshes smaller than a tile,
one cell short of it, exactly one and one cell past it (tiles are 8 x 8 and
4 x 4 x 4 cells for the table stage, the pseudo-step and the limiter, 8 to 32
cells wide for the separable stage), one-cell axes, every basis and degree.

FP64 against the oracle: the same quadratures in another association, so 1e-12
of the largest entry for one evaluation and 1e-11 after a sweep.

FP32 against FP64 from the same 32-bit coefficients: a coefficient of the rate
is a sum of products (velocity) x (field value) x (modal factor)/h.  The modal
factors of one axis are at most (2p+1)^(1/2) per value and (2p+1)^(3/2) per
derivative, their sum over the modes at most (p+1)^3 for each axis it is taken
over, and a value passes through fewer than 60 roundings of 2^-24 on its way
(three axes, two sums per axis, the lifts and the combination)."""
import ctypes as C

import numpy as np
import pytest

from felspa_b200 import abi, fields as F
from felspa_b200.batch import Batch
from felspa_b200.learned import MLP, param_layout, split_params
from felspa_b200.level_set import AdvectSimulator, Mesh, Problem, ReinitSimulatorLDG, dealii_hypercube_order
from felspa_b200.lib import FlspError, check, load

pytestmark = pytest.mark.gpu

Q, P = abi.BASIS_Q, abi.BASIS_P
SPACES = [(2, 1, P), (2, 1, Q), (2, 2, P), (2, 2, Q), (2, 3, P), (2, 3, Q), (3, 1, P), (3, 1, Q), (3, 2, P), (3, 2, Q)]
MESHES = {2: [(1, 1), (7, 9), (8, 8), (33, 1), (17, 16)], 3: [(1, 1, 1), (3, 5, 4), (4, 4, 4), (9, 1, 8), (8, 9, 5)]}
CASES = [(p, b, n) for dim, p, b in SPACES for n in MESHES[dim]]


def rel(a, b):
    return float(np.max(np.abs(a - b)) / max(np.max(np.abs(b)), 1e-300))


def velocity(dim, table):
    """one separable term per component, or a sum of terms (tabulated)"""
    base = F.single_vortex(period=2.0) if dim == 2 else F.deformation_3d()
    if not table:
        return base
    drift = F.constant((0.3, -0.2, 0.1)[:dim])
    return F.VelocityField(dim, base.terms + drift.terms, time_kind=base.time_kind, ta=base.ta, tb=base.tb)


def coefficients(n_dofs, nb, seed):
    """a field that is rough (both upwind sides and signs occur in every tile)"""
    v = np.random.default_rng(seed).standard_normal((n_dofs // nb, nb))
    v[:, 1:] *= 0.3
    return v.astype(np.float32).astype(np.float64).ravel()


# (degree 1, total-degree basis, one cell, no drift: the rate is identically zero,
# so nothing to be relative to)
STAGE = [c + (t,) for c in CASES for t in (False, True) if t or c[:2] != (1, P) or max(c[2]) > 1]


@pytest.mark.parametrize("p,basis,n,table", STAGE)
def test_stage(oracle, flsp, p, basis, n, table):
    dim = len(n)
    field = velocity(dim, table)
    orc = oracle.Problem(dim, n, p, basis)
    orc.set_velocity(field)
    phi = coefficients(orc.n_dofs, orc.nb, 3)
    want = orc.advect_rhs(phi, 0.3)
    for prec in (abi.FP64, abi.FP32):
        pb = Problem(Mesh(dim, n), p, basis=basis, precision=prec)
        pb.set_velocity(field)
        pb.set_state(phi)
        got = np.empty(pb.n_dofs)
        check(load().flsp_advect_rhs(pb.h, 0.3, got.ctypes.data_as(C.POINTER(C.c_double)), got.size))
        if prec == abi.FP64:
            assert rel(got, want) <= 1e-12
        else:
            umax = 3.0 if dim == 2 else 2.5
            bound = 60 * 2.0 ** -24 * (2 * p + 1) ** 1.5 * (p + 1) ** 3 * umax * max(n) * np.max(np.abs(phi))
            assert np.max(np.abs(got - want)) <= bound
        pb.close()


@pytest.mark.parametrize("p,basis,n", CASES)
def test_sweep(oracle, flsp, p, basis, n):
    """gradients, then two pseudo-steps (2D with viscosity: the diffusion too)"""
    dim = len(n)
    orc = oracle.Problem(dim, n, p, basis)
    phi = orc.project(F.sphere((0.47, 0.56, 0.52)[:dim], 0.31))
    sim = AdvectSimulator(Mesh(dim, n), p, basis=basis, precision=abi.FP64)
    sim.problem.set_state(phi)
    reinit = ReinitSimulatorLDG(sim.problem)
    for got, want in zip(reinit.local_left_right_gradients(), orc.hj_gradients(phi)):
        assert rel(got, want) <= 1e-12
    o = abi.default_reinit_opts(mode=abi.REINIT_FIXED, n_pseudo_steps=2, limiter=0,
                                viscosity=1e-3 if dim == 2 else 0.0)
    reinit.run_iteration(o)
    st, _ = orc.reinit(phi, o)
    assert st == 0
    assert rel(sim.get_solution_vector(), phi) <= 1e-11


@pytest.mark.parametrize("p,basis,n", [c for c in CASES if len(c[2]) == 3] + [(2, Q, (1, 5)), (2, P, (18, 2)),
                                                                          (3, Q, (35, 9))])
def test_viscous_sweep(oracle, flsp, p, basis, n):
    """the diffusion term reads two cells to each side: axes of one, two and
    more cells, blocks (16 x 8, 4 x 4 x 4) that end in the mesh"""
    dim = len(n)
    orc = oracle.Problem(dim, n, p, basis)
    phi = orc.project(F.sphere((0.47, 0.56, 0.52)[:dim], 0.31))
    pb = Problem(Mesh(dim, n), p, basis=basis, precision=abi.FP64)
    pb.set_state(phi)
    o = abi.default_reinit_opts(mode=abi.REINIT_FIXED, n_pseudo_steps=3, limiter=0, viscosity=5e-3, cfl_max=0.1)
    ReinitSimulatorLDG(pb).run_iteration(o)
    st, _ = orc.reinit(phi, o)
    assert st == 0
    assert rel(pb.get_state(), phi) <= 1e-11
    pb.close()


@pytest.mark.parametrize("p,basis,n", [c for c in CASES if len(c[2]) == 2])
def test_limiter(oracle, flsp, p, basis, n):
    """the rough field: nearly every cell is troubled"""
    orc = oracle.Problem(2, n, p, basis)
    phi = coefficients(orc.n_dofs, orc.nb, 5)
    pb = Problem(Mesh(2, n), p, basis=basis, precision=abi.FP64)
    pb.set_state(phi)
    assert ReinitSimulatorLDG(pb).apply_weno_limiter() == orc.weno(phi)
    assert rel(pb.get_state(), phi) <= 1e-11
    pb.close()


@pytest.mark.parametrize("n", [(33, 20), (9, 7, 10)])
def test_band_over_everything_p_basis(flsp, n):
    """the band's tile lists (launch tiles of several blocks) against the full sweep"""
    dim = len(n)
    outs = []
    for kw in ({}, {"narrow_band": 1, "band_cells": 1e9}):
        pb = Problem(Mesh(dim, n), 2, basis=P, precision=abi.FP64)
        pb.project(F.sphere((0.47, 0.56, 0.52)[:dim], 0.31))
        ReinitSimulatorLDG(pb).run_iteration(
            abi.default_reinit_opts(mode=abi.REINIT_FIXED, n_pseudo_steps=3, **kw))
        outs.append(pb.get_state())
        pb.close()
    assert np.array_equal(outs[0], outs[1])


@pytest.mark.parametrize("p,basis,n", [(2, P, (33, 20)), (3, Q, (17, 9)), (1, P, (9, 7, 10)), (2, Q, (9, 7, 10))])
def test_viscous_band_over_everything(flsp, p, basis, n):
    """the diffusion term with every band tile listed is the full sweep's"""
    dim = len(n)
    outs = []
    for kw in ({}, {"narrow_band": 1, "band_cells": 1e9}):
        pb = Problem(Mesh(dim, n), p, basis=basis, precision=abi.FP64)
        pb.project(F.sphere((0.47, 0.56, 0.52)[:dim], 0.31))
        ReinitSimulatorLDG(pb).run_iteration(abi.default_reinit_opts(
            mode=abi.REINIT_FIXED, n_pseudo_steps=3, viscosity=5e-3, cfl_max=0.1, limiter=0, **kw))
        outs.append(pb.get_state())
        pb.close()
    assert np.array_equal(outs[0], outs[1])


@pytest.mark.parametrize("steps", [1, 31, 32, 33, 70])
def test_substeps_ahead(flsp, steps):
    """substeps computed up to 32 ahead equal substeps computed one by one"""
    outs = []
    for chunk in (steps, 1):
        sim = AdvectSimulator(Mesh(2, (9, 12)), 2, basis=Q, precision=abi.FP64, cfl_max=0.1)
        sim.initialize(F.sphere((0.4, 0.6), 0.2), F.single_vortex(period=0.5))
        for _ in range(steps // chunk):
            sim.advance_steps(chunk)
        outs.append((sim.get_solution_vector(), sim.get_time(), sim.problem.get_step_count()))
    assert np.array_equal(outs[0][0], outs[1][0]) and outs[0][1:] == outs[1][1:]
    assert outs[0][2] == steps


@pytest.mark.parametrize("prec", [abi.FP64, abi.FP32])
def test_batch_members(flsp, prec):
    """members one cell around the tile, every degree: each as it runs alone"""
    shapes = [(7, 9), (8, 8), (9, 7), (1, 17), (16, 16), (15, 33)]
    field = velocity(2, True)
    ctl = abi.default_ls_opts(reinit_frequency=4, reinit=abi.default_reinit_opts(mode=abi.REINIT_FIXED,
                                                                                 n_pseudo_steps=2))
    for p in (1, 2, 3):
        b = Batch([Mesh(2, n) for n in shapes], [p] * len(shapes), precision=prec, cfl_max=0.1)
        singles = []
        for pb, n in zip(b.problems, shapes):
            one = Problem(Mesh(2, n), p, basis=Q, precision=prec, cfl_max=0.1)
            singles.append(one)
            for x in (pb, one):
                x.set_velocity(field)
                x.project(F.sphere((0.4927, 0.5481), 0.27))
        b.run_steps(9, ctl)
        for pb, one in zip(b.problems, singles):
            check(load().flsp_ls_run_steps(one.h, C.byref(ctl), 9))
            one.sync()
            assert rel(pb.get_state(), one.get_state()) <= (1e-12 if prec == abi.FP64 else 1e-4)
            one.close()
        b.close()


@pytest.mark.parametrize("prec", [abi.FP64, abi.FP32])
@pytest.mark.parametrize("ordered", [False, True])
def test_state_checked_on_the_device(flsp, prec, ordered):
    """both ways a state takes (copied as it is, or converted / permuted):
    round trip, count of the values that are not finite, and a good state after"""
    mesh = Mesh(2, (8, 8), host_cell_order=dealii_hypercube_order(2, 2, 2) if ordered else None)
    pb = Problem(mesh, 2, basis=Q, precision=prec)
    good = coefficients(pb.n_dofs, 9, 7)
    pb.set_state(good)
    assert np.array_equal(pb.get_state(), good)
    bad = good.copy()
    bad[[0, 17, -1]] = [np.inf, np.nan, -np.inf]
    with pytest.raises(FlspError, match="3 non-finite"):
        pb.set_state(bad)
    pb.set_state(good)
    assert np.array_equal(pb.get_state(), good)
    pb.close()


def test_rejected_lattice_leaves_the_velocity(flsp):
    n = (6, 5)
    sim = AdvectSimulator(Mesh(2, n), 2, basis=Q, precision=abi.FP64, cfl_max=0.1)
    sim.initialize(F.sphere((0.4, 0.6), 0.2), F.single_vortex())
    bad = F.random_fe_lattice(n, 2, seed=1).copy()
    bad.ravel()[-1] = np.nan
    for good in (None, F.random_fe_lattice(n, 2, seed=2), F.random_fe_lattice(n, 1, seed=3)):
        if good is not None:
            sim.problem.set_velocity_fe(1 if good.size < bad.size else 2, good)
        before = sim.explicit_time_derivative(0.2)
        with pytest.raises(FlspError, match="non-finite"):
            sim.problem.set_velocity_fe(2, bad)
        assert np.array_equal(sim.explicit_time_derivative(0.2), before)


@pytest.mark.parametrize("dim", [2, 3])
def test_network_row_edges(flsp, oracle, dim):
    """batches around the 128-row tile, after a larger and before a smaller one
    in the same kept buffers; bf16 operands: bounds of the network's other
    tests (2e-2 of the largest output, 3e-2 relative Frobenius per gradient)"""
    torch = pytest.importorskip("torch")

    def bf16(a):
        return torch.tensor(np.asarray(a, dtype=np.float32)).to(torch.bfloat16).float().numpy().astype(np.float64)

    rng = np.random.default_rng(31)
    par = np.concatenate([(rng.uniform(-1.5, 1.5, size=s) / np.sqrt(s[1]) if name.startswith("W")
                           else rng.uniform(-0.1, 0.1, size=s)).ravel()
                          for name, _, s in param_layout(dim)]).astype(np.float32)
    v = split_params(par.astype(np.float64), dim)
    Ws, bs = [bf16(v[f"W{l}"]) for l in range(1, 6)], [v[f"b{l}"].copy() for l in range(1, 6)]
    net = MLP(device=0, seed=1, dim=dim)
    net.set_params(par)
    for rows in (257, 1, 127, 128, 129):
        x = rng.standard_normal((rows, net.n_in)).astype(np.float32)
        dy = (rng.standard_normal((rows, net.n_out)) / rows).astype(np.float32)
        ref = oracle.mlp_forward(Ws, bs, bf16(x))
        assert np.max(np.abs(net.forward(x) - ref)) <= 2e-2 * np.max(np.abs(ref))
        dW, db = oracle.mlp_backward(Ws, bs, bf16(x), bf16(dy))
        g = split_params(net.backward(x, dy).astype(np.float64), dim)
        for l in range(5):
            for got, want in ((g[f"W{l + 1}"], dW[l]), (g[f"b{l + 1}"], db[l])):
                assert np.linalg.norm(got - want) <= 3e-2 * np.linalg.norm(want)
    net.close()
