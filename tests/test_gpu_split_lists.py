"""The split stepper's force kernels on long and on ragged lists of poses, against the fused stepper.

Both sum every pose's terms in the same order, so after the same steps the poses of all trajectories are
equal bit for bit, and so are the numbers of stencils and far-field evaluations, which do not depend on
how poses are spread over warps.  Sizes follow from the warps that are resident on the device.
"""

import dataclasses

import numpy as np
import pytest

from tests.helpers import system
from tests.test_gpu_stepper import make_sim

pytestmark = pytest.mark.gpu

COUNTS = ("steps", "returns", "overlap", "grid_evals", "ff_evals", "rev_evals")


def _sms():
    import torch

    return torch.cuda.get_device_properties(0).multi_processor_count


def _after(s, n, steps, precision, torque, group, **kw):
    """Every trajectory's pose and the counters after `steps` steps of one launch."""
    from pystarc_b200 import _lib

    sim = make_sim(s, n, 1_000_000, precision, torque, slots=n, steps_per_launch=steps, launches_per_poll=1, **kw)
    h = sim.engine.handle
    h.call("bd_set_launch", group, 128)
    sim._setup()
    h.call("bd_sim_reset", None)
    h.call("bd_sim_run", 1, steps, None)
    c, q = np.zeros(3 * n), np.zeros(4 * n)
    traj, nstep, rets = (np.zeros(n, dtype=np.int32) for _ in range(3))
    status, live, ctr = np.zeros(n, dtype=np.int8), _lib.C.c_int32(), np.zeros(_lib.N_CTR, dtype=np.uint64)
    i32 = _lib.C.c_int32
    h.call("bd_sim_snapshot", _lib.ptr(c), _lib.ptr(q), _lib.ptr(traj, i32), _lib.ptr(nstep, i32), _lib.ptr(rets, i32),
           _lib.ptr(status, _lib.C.c_int8), _lib.C.byref(live), _lib.ptr(ctr, _lib.C.c_uint64))
    counters = sim.read_counters()
    sim.engine.close()
    m = live.value
    order = np.argsort(traj[:m])
    rows = np.concatenate([c.reshape(3, n)[:, :m], q.reshape(4, n)[:, :m], nstep[None, :m], rets[None, :m]])
    return rows[:, order], {k: counters[k] for k in COUNTS}


def _assert_same(s, n, steps, precision, torque, **kw):
    a, ca = _after(s, n, steps, precision, torque, 65, **kw)
    b, cb = _after(s, n, steps, precision, torque, 66, **kw)
    np.testing.assert_array_equal(a, b)
    assert ca == cb


# four poses share a warp in mixed precision above four poses for each of 16 warps per SM
@pytest.mark.parametrize("n_of", [lambda w: 4 * w + 1, lambda w: 4 * w + 3, lambda w: 17 * w - 253])
@pytest.mark.parametrize("torque", ["zero", "centroid"])
def test_four_small_ligands_share_a_warp(n_of, torque):
    s = dataclasses.replace(system("c2"), r_start=14.0, r_escape=40.0)  # some poses near, some far
    _assert_same(s, n_of(16 * _sms()), 4, "mixed", torque)


# a warp takes several entries a turn from 16 poses per warp on: 16 at most, 512 atoms of larger ligands
@pytest.mark.parametrize("n_of", [lambda w: 16 * w - 1, lambda w: 16 * w, lambda w: 25 * w + 5, lambda w: 130 * w + 7])
@pytest.mark.parametrize("atoms", [18, 90])
def test_a_warp_takes_several_poses_a_turn(n_of, atoms):
    from pystarc_b200 import synth

    if atoms == 18:
        s = dataclasses.replace(system("c2"), r_start=14.0, r_escape=40.0, lig_born_grids=[])
    else:
        s = dataclasses.replace(synth.config3(scale=0.4, device="cuda"), r_start=20.0, r_escape=60.0, lig_born_grids=[])
    assert len(s.lig_q) >= atoms
    _assert_same(s, n_of(16 * _sms()), 3, "fp64" if atoms == 18 else "mixed", "centroid")
