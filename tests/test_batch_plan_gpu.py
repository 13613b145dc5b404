"""A batch whose members change between runs: every run steps each member as the
problem alone would step."""
import ctypes as C

import numpy as np
import pytest

from felspa_b200 import abi, fields as F
from felspa_b200.batch import Batch
from felspa_b200.level_set import Mesh, Problem
from felspa_b200.lib import FlspError, check, load

pytestmark = pytest.mark.gpu

CTL = abi.default_ls_opts(reinit_frequency=4, reinit=abi.default_reinit_opts(mode=abi.REINIT_FIXED, n_pseudo_steps=2))


def test_velocity_set_again(flsp):
    """another field with another time factor for one member, then for every
    member, between runs that replay and runs that end inside a period"""
    shapes = [(7, 9), (16, 16), (12, 20)]
    still, vortex, fast = F.ccw_rotation(), F.single_vortex(period=0.7), F.single_vortex(period=0.3)
    b = Batch([Mesh(2, n) for n in shapes], [1, 2, 3], precision=abi.FP64, cfl_max=0.1)
    singles = [Problem(Mesh(2, n), p, basis=abi.BASIS_Q, precision=abi.FP64, cfl_max=0.1)
               for n, p in zip(shapes, (1, 2, 3))]
    for x in b.problems + singles:
        x.project(F.sphere((0.4927, 0.5481), 0.27))
    for velocities, steps in (([still] * 3, 9), ([still, vortex, still], 7), ([fast, vortex, fast], 8),
                              ([vortex, still, fast], 4)):
        for pb, one, v in zip(b.problems, singles, velocities):
            pb.set_velocity(v)
            one.set_velocity(v)
        b.run_steps(steps, CTL)
        for pb, one in zip(b.problems, singles):
            check(load().flsp_ls_run_steps(one.h, C.byref(CTL), steps))
            one.sync()
            assert abs(pb.get_time() - one.get_time()) <= 1e-14
            a, r = pb.get_state(), one.get_state()
            assert np.max(np.abs(a - r)) <= 1e-12 * np.max(np.abs(r))
    for one in singles:
        one.close()
    b.close()


def test_velocity_missing(flsp):
    b = Batch([Mesh(2, (8, 8))] * 2, [1, 2], precision=abi.FP64, cfl_max=0.1)
    b.problems[0].set_velocity(F.ccw_rotation())
    with pytest.raises(FlspError, match="velocity not set"):
        b.run_steps(1, CTL)
    b.problems[1].set_velocity(F.ccw_rotation())
    b.run_steps(1, CTL)
    b.close()
