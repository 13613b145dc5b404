"""The 32-bit reinitialisation, limiter and batch kernels at the edges of their
tiles, against the 64-bit oracle from the same 32-bit coefficients.

Tolerance: every sum a kernel forms is over values of at most V, the largest
sum over a cell's modes of |coefficient| max |mode|, and a result passes through
fewer than ROUNDINGS roundings on its way.  One rounding of 2^-24 of V at the
input of a sum is what a change of the coefficients by 2^-24 V is, and what that
does to the result the oracle says: the largest change over DRAWS random
changes (one sign per coefficient), times ROUNDINGS, per operator applied."""
import ctypes as C

import numpy as np
import pytest

from felspa_b200 import abi, fields as F
from felspa_b200.batch import Batch
from felspa_b200.level_set import Mesh, Problem, ReinitSimulatorLDG

pytestmark = pytest.mark.gpu

Q, P = abi.BASIS_Q, abi.BASIS_P
ROUNDINGS, DRAWS = 60, 8
SWEEPS = [(p, b, n) for p in (1, 2, 3) for b in (Q, P) for n in ((7, 9), (17, 16), (33, 1))] + \
         [(p, b, n) for p in (1, 2) for b in (Q, P) for n in ((3, 5, 4), (9, 7, 10), (17, 9, 6))]
BALL = F.sphere((0.47, 0.56, 0.52), 0.31)


def modes(dim, p, basis):
    r = range(p + 1)
    every = [(a, b, c) for c in (r if dim == 3 else (0,)) for b in r for a in r]
    return [m for m in every if basis == Q or sum(m) <= p]


def ball(dim):
    return BALL if dim == 3 else F.sphere((0.47, 0.56), 0.31)


def rounded(orc):
    return orc.project(ball(orc.dim)).astype(np.float32).astype(np.float64)


def size_of(phi, dim, p, basis):
    """V: |L_a| <= L_a(1) = sqrt(2a + 1)"""
    w = np.array([np.prod(np.sqrt(2.0 * np.array(m) + 1.0)) for m in modes(dim, p, basis)])
    return float((np.abs(phi).reshape(-1, w.size) @ w).max())


def reach(op, phi, V, seed=1):
    """what a rounding at the inputs does to op's result, per entry's largest"""
    rng = np.random.default_rng(seed)
    at = op(phi)
    return at, max(float(np.max(np.abs(op(phi + 2.0 ** -24 * V * rng.choice([-1.0, 1.0], phi.size)) - at)))
                   for _ in range(DRAWS))


def swept(prec, n, p, basis, phi, o):
    pb = Problem(Mesh(len(n), n), p, basis=basis, precision=prec)
    pb.set_state(phi)
    ReinitSimulatorLDG(pb).run_iteration(o)
    out = pb.get_state()
    pb.close()
    return out


@pytest.mark.parametrize("visc", [0.0, 5e-3])
@pytest.mark.parametrize("p,basis,n", SWEEPS)
def test_pseudo_step(oracle, flsp, p, basis, n, visc):
    dim = len(n)
    orc = oracle.Problem(dim, n, p, basis)
    phi = rounded(orc)
    o = abi.default_reinit_opts(mode=abi.REINIT_FIXED, n_pseudo_steps=1, limiter=0, viscosity=visc,
                                cfl_max=0.1 if visc else 0.2)

    def op(x):
        x = x.copy()
        assert orc.reinit(x, o)[0] == 0
        return x
    want, change = reach(op, phi, size_of(phi, dim, p, basis))
    # the sign table, the step (with viscosity, the diffusion term before it)
    assert np.max(np.abs(swept(abi.FP32, n, p, basis, phi, o) - want)) <= (3 if visc else 2) * ROUNDINGS * change


@pytest.mark.parametrize("visc", [0.0, 5e-3])
@pytest.mark.parametrize("p,basis,n", [(2, P, (9, 7, 10)), (2, P, (17, 9, 6)), (1, P, (17, 9, 6)), (2, Q, (9, 7, 10)),
                                       (2, P, (33, 20)), (3, Q, (17, 9))])
def test_band_over_everything(flsp, p, basis, n, visc):
    """the band's tile lists (P basis: launch tiles of two blocks at 3D degree
    2, of several in 2D) are the full sweep to the last bit"""
    pb = Problem(Mesh(len(n), n), p, basis=basis, precision=abi.FP32)
    pb.project(ball(len(n)))
    phi = pb.get_state()
    pb.close()
    kw = dict(mode=abi.REINIT_FIXED, n_pseudo_steps=3, limiter=0, viscosity=visc, cfl_max=0.1)
    full = swept(abi.FP32, n, p, basis, phi, abi.default_reinit_opts(**kw))
    assert np.array_equal(full, swept(abi.FP32, n, p, basis, phi,
                                      abi.default_reinit_opts(narrow_band=1, band_cells=1e9, **kw)))


@pytest.mark.parametrize("p,basis,n", [(2, P, (9, 7, 10)), (2, P, (17, 9, 6)), (2, P, (30, 26, 28)), (1, P, (17, 9, 6)),
                                       (2, Q, (9, 7, 10)), (2, P, (40, 36))])
def test_band_of_a_few_cells(oracle, flsp, p, basis, n):
    """the same coefficients give FP32 and FP64 the same band (a cell mean is a
    coefficient, compared in 64 bits): cells outside it keep every bit, cells in
    it take the step.  A threshold on a cell mean itself is taken too."""
    dim = len(n)
    orc = oracle.Problem(dim, n, p, basis)
    phi = rounded(orc)
    cells = phi.reshape(-1, orc.nb)
    diam = Mesh(dim, n).min_diameter
    rhs = orc.hj_rhs(phi, phi)
    means = np.sort(np.abs(cells[:, 0]))
    for band in (1.0, float(means[means.size // 3] / diam)):
        o = abi.default_reinit_opts(mode=abi.REINIT_FIXED, n_pseudo_steps=1, limiter=0, narrow_band=1, band_cells=band)
        inside = np.abs(cells[:, 0]) <= band * diam
        assert inside.any() and not inside.all()
        got, want = (swept(x, n, p, basis, phi, o).reshape(cells.shape) for x in (abi.FP32, abi.FP64))
        for s in (got, want):
            assert np.array_equal(s[~inside], cells[~inside])
        # the step's size in FP64, and the change of phi + dt rhs
        r = rhs.reshape(cells.shape)[inside]
        dt = float(np.sum((want - cells)[inside] * r) / np.sum(r * r))
        _, change = reach(lambda x: x + dt * orc.hj_rhs(x, x), phi, size_of(phi, dim, p, basis))
        assert np.max(np.abs(got - want)) <= 2 * ROUNDINGS * change


@pytest.mark.parametrize("rough", [True, False])
@pytest.mark.parametrize("p,basis,n", [(p, b, n) for p in (1, 2, 3) for b in (Q, P) for n in ((7, 9), (17, 16), (33, 2))])
def test_limiter(oracle, flsp, p, basis, n, rough):
    """cells whose detector is decided by more than the roundings: the others
    may go either way"""
    orc = oracle.Problem(2, n, p, basis)
    phi = rounded(orc)
    if rough:
        v = np.random.default_rng(5).standard_normal((phi.size // orc.nb, orc.nb))
        v[:, 1:] *= 0.3
        phi = v.astype(np.float32).astype(np.float64).ravel()
    V = size_of(phi, 2, p, basis)
    ms = modes(2, p, basis)
    c = phi.reshape(n[1], n[0], orc.nb)
    mean = c[..., 0]
    tau = ROUNDINGS * 2.0 ** -24 * V
    sure = np.zeros((n[1], n[0]), dtype=bool)          # surely troubled
    fine = np.ones((n[1], n[0]), dtype=bool)           # surely not
    pad = np.pad(mean, 1, constant_values=np.nan)
    for vy in (0, 1):
        for vx in (0, 1):
            w = np.array([np.sqrt(2 * a + 1) * (1 if vx else (-1) ** a) * np.sqrt(2 * b + 1) * (1 if vy else (-1) ** b)
                          for a, b, _ in ms])
            a = c @ w - mean
            d = 1.5 * (pad[1:-1, 2:] - mean if vx else pad[1:-1, :-2] - mean)
            d = d + 1.5 * (pad[2:, 1:-1] - mean if vy else pad[:-2, 1:-1] - mean)
            use = ~np.isnan(d)
            d = np.where(use, d, 0.0)
            # mm = a when the signs agree and |a| <= |d|, else 0 or |d|
            big = (np.abs(a) > tau) & ((np.abs(a) > np.abs(d) + 4 * tau) | ((a * d < 0) & (np.abs(d) > 4 * tau)))
            ok = (a * d > 0) & (np.abs(d) > np.abs(a) + 4 * tau)
            sure |= use & big
            fine &= ~use | ok
    sure, fine = sure.ravel(), fine.ravel()
    flags = orc.minmod_flags(phi).astype(bool)
    assert np.all(flags[sure]) and not np.any(flags[fine])
    assert (sure if rough else sure | fine).mean() > 0.5

    def op(x):
        x = x.copy()
        orc.weno(x)
        return x
    want = op(phi)
    rng = np.random.default_rng(1)
    change = 0.0
    for _ in range(DRAWS):
        x = op(phi + 2.0 ** -24 * V * rng.choice([-1.0, 1.0], phi.size))
        change = max(change, float(np.max(np.abs(x - want).reshape(-1, orc.nb)[sure | fine], initial=0.0)))
    pb = Problem(Mesh(2, n), p, basis=basis, precision=abi.FP32)
    pb.set_state(phi)
    ReinitSimulatorLDG(pb).apply_weno_limiter()
    got = pb.get_state().reshape(-1, orc.nb)
    pb.close()
    assert np.array_equal(got[fine], phi.reshape(-1, orc.nb)[fine])
    if sure.any():
        assert np.max(np.abs(got - want.reshape(-1, orc.nb))[sure]) <= ROUNDINGS * change


@pytest.mark.parametrize("prec", [abi.FP64, abi.FP32])
def test_batch_members_against_the_oracle(oracle, flsp, prec):
    """four substeps and a sweep of two pseudo-steps of every member"""
    shapes = [(7, 9), (16, 16), (9, 17), (1, 12)]
    base, drift = F.single_vortex(period=2.0), F.constant((0.3, -0.2))
    field = F.VelocityField(2, base.terms + drift.terms, time_kind=base.time_kind, ta=base.ta, tb=base.tb)
    ctl = abi.default_ls_opts(reinit_frequency=4, reinit=abi.default_reinit_opts(mode=abi.REINIT_FIXED,
                                                                                 n_pseudo_steps=2, limiter=0))
    for p in (1, 2, 3):
        b = Batch([Mesh(2, n) for n in shapes], [p] * len(shapes), precision=prec, cfl_max=0.1)
        starts = []
        for pb, n in zip(b.problems, shapes):
            starts.append(rounded(oracle.Problem(2, n, p, Q)))
            pb.set_velocity(field)
            pb.set_state(starts[-1])
        b.run_steps(4, ctl)
        for pb, n, phi in zip(b.problems, shapes, starts):
            def op(x):
                orc = oracle.Problem(2, n, p, Q)
                orc.set_velocity(field)
                x = x.copy()
                for _ in range(4):
                    orc.ls_advance(x, 1e9, ctl, single_step=True, cfl_max=0.1)
                return x
            want, change = reach(op, phi, size_of(phi, 2, p, Q))
            err = np.max(np.abs(pb.get_state() - want))
            if prec == abi.FP64:
                assert err <= 1e-11 * np.max(np.abs(want))
            else:   # twelve stages, the sign table, two pseudo-steps
                assert err <= 15 * ROUNDINGS * change
        b.close()
