"""A kernel whose wait for its bulk copies runs out sets the problem's error word
and returns; the call that computed with it reports FLSP_ERR_TIMEOUT instead of a
result.  The word is set from the host here (flsp_set_device_error)."""
import ctypes as C

import numpy as np
import pytest

from felspa_b200 import abi, fields as F
from felspa_b200.learned import MLP, default_learned_opts
from felspa_b200.level_set import LevelSetSurface, Mesh, ReinitSimulatorLDG
from felspa_b200.lib import FlspError, check, load

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [abi.FP64, abi.FP32])
@pytest.mark.parametrize("n", [(16, 12), (6, 5, 4)])
def test_results_of_a_failed_wait_are_not_returned(flsp, prec, n):
    dim = len(n)
    fixed = abi.default_reinit_opts(mode=abi.REINIT_FIXED, n_pseudo_steps=2)
    ls = LevelSetSurface(Mesh(dim, n), 2, basis=abi.BASIS_Q, precision=prec, cfl_max=0.1,
                         control=abi.default_ls_opts(reinit_frequency=2, reinit=fixed))
    ls.initialize(F.sphere((0.4927, 0.5481, 0.51)[:dim], 0.27), F.single_vortex() if dim == 2 else F.deformation_3d())
    pb, reinit = ls.problem, ReinitSimulatorLDG(ls.problem)
    calls = [lambda: ls.explicit_time_derivative(0.2), lambda: reinit.run_iteration(fixed),
             lambda: reinit.run_iteration(abi.default_reinit_opts(mode=abi.REINIT_BAND)),
             lambda: ls.advance_time(1.0, True), lambda: ls.advance_steps(2), lambda: ls.run_steps(3)]
    if dim == 2:
        calls.append(reinit.apply_weno_limiter)
    for call in calls:
        check(load().flsp_set_device_error(pb.h, 1))
        with pytest.raises(FlspError, match="ran out"):
            call()
        check(load().flsp_set_device_error(pb.h, 0))
        call()
    assert np.all(np.isfinite(pb.get_state()))


def test_learned_sweep(flsp):
    """the fallback sweep of a learned reinitialisation, and the pairs of a collection"""
    ls = LevelSetSurface(Mesh(2, (24, 24)), 2, basis=abi.BASIS_Q, precision=abi.FP32, cfl_max=0.1)
    ls.initialize(F.sphere((0.4927, 0.5481), 0.27), F.single_vortex())
    net = MLP(device=0, seed=3)
    check(load().flsp_set_device_error(ls.problem.h, 1))
    with pytest.raises(FlspError, match="ran out"):
        net.reinit(ls.problem, default_learned_opts(max_residual=1e-12))
    with pytest.raises(FlspError, match="ran out"):
        net.collect(ls.problem, band_cells=6.0)
    check(load().flsp_set_device_error(ls.problem.h, 0))
    n = net.collect(ls.problem, band_cells=6.0)
    assert n > 0
    net.close()
