"""How an SSP-RK3 stage combines with phi^n, to the last bit.

A narrow band and a learned reinitialisation compare cell means with a
threshold, so the result of such a run is a step function of the last bits of
the field.  In FP32, where a mean is near enough to the threshold for that to
happen, the combination keeps the reference's operation order,
((phi_2 + dt L) 2 + phi^n) (1/3) for the last stage
(time_integration.implement.h:141-234); FP64 adds a share of the difference to
phi^n, which does not scale the field.

A constant field in a uniform flow shows it alone: the two fluxes of a cell are
the same numbers, so L has no mean and the mean of a cell follows the
combination's roundings, away from the ends by more than the three cells a step
that a boundary reaches."""
import numpy as np
import pytest

from felspa_b200 import abi, fields as F
from felspa_b200.level_set import LevelSetSurface, Mesh

pytestmark = pytest.mark.gpu

STEPS = 4


def flow(dim, terms):
    """along x; one term (separable stage kernel) or a sum of two (tabulated)"""
    zero = [0.0] * (dim - 1)
    if terms == 1:
        return F.constant((0.7, *zero))
    a, b = F.constant((0.4, *zero)), F.constant((0.3, *zero))
    return F.VelocityField(dim, a.terms + b.terms)


def mean_after(c, T):
    """L = 0: the stages before the last give the mean back exactly (4 c / 4)"""
    m = T(c)
    if T is np.float64:
        return m   # m + w (m - m)
    for _ in range(STEPS):
        m = T(T(T(2) * m + m) * (T(1) / T(3)))
    return m


@pytest.mark.parametrize("prec", [abi.FP32, abi.FP64])
@pytest.mark.parametrize("n,p,basis,terms", [
    ((40, 9), 2, abi.BASIS_Q, 1), ((40, 9), 1, abi.BASIS_P, 1), ((40, 9), 3, abi.BASIS_Q, 2),
    ((40, 3, 3), 2, abi.BASIS_P, 1), ((40, 5, 4), 2, abi.BASIS_Q, 1), ((40, 3, 3), 2, abi.BASIS_P, 2),
    ((40, 4, 4), 1, abi.BASIS_Q, 2)])
def test_means_follow_the_combination(flsp, prec, n, p, basis, terms):
    T = np.float32 if prec == abi.FP32 else np.float64
    assert (mean_after(0.83, T) != T(0.83)) == (prec == abi.FP32)   # the value shows the order
    ctl = abi.default_ls_opts(reinit_frequency=1000, reinit=abi.default_reinit_opts(
        mode=abi.REINIT_FIXED, n_pseudo_steps=2, narrow_band=1, band_cells=6.0))
    for c in (0.83, 0.1, 0.7):
        ls = LevelSetSurface(Mesh(len(n), n), p, basis=basis, precision=prec, cfl_max=0.1, control=ctl)
        ls.problem.set_velocity(flow(len(n), terms))
        phi = np.zeros(ls.n_dofs)
        nb = ls.n_dofs // int(np.prod(n))
        phi[::nb] = T(c)
        for run in (ls.run_steps, ls.advance_steps):
            ls.problem.set_state(phi)
            run(STEPS)
            means = ls.get_solution_vector()[::nb].reshape(n[::-1])
            assert np.all(means[..., 3 * STEPS:n[0] - 3 * STEPS] == mean_after(c, T))
