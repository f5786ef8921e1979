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


@pytest.mark.parametrize("precision,torque,per_sm", [("fp64", "zero", 16), ("fp64", "centroid", 16),
                                                     ("mixed", "zero", 32), ("mixed", "centroid", 24)])
@pytest.mark.parametrize("sysname", ["c2_full", "c3_full"])
def test_poses_in_contact_shared_among_warps(sysname, precision, torque, per_sm):
    """All poses near contact on receptors of 54 and 101 chunks: eight, four and two warps share a pose of
    the sweep, drain in the middle of it and take several rounds; then one warp a pose, several each."""
    from pystarc_b200 import synth

    if sysname == "c2_full":
        s = dataclasses.replace(synth.config2(device="cuda"), r_start=26.0, r_escape=80.0)
    else:
        s = dataclasses.replace(synth.config3(device="cuda"), r_start=30.0, r_escape=90.0)
    w = per_sm * _sms()  # resident warps of the sweep
    sizes = [w // 4 - 1, w // 2, w - 3, 2 * w + 5] if sysname == "c2_full" else [w // 4, w // 2 - 1, w // 2 + 60]
    for n in sizes:
        _assert_same(s, n, 3, precision, torque)


def _batch_equals_alone(systems, n, steps, precision, torque):
    """Fates and evaluation counts (which follow from every pose) of a batch are those of its systems alone."""
    from pystarc_b200.multi import B200MultiBatch

    kw = dict(steps_per_launch=5, launches_per_poll=2)
    sims = [make_sim(s, n + 7 * i, steps, precision, torque, seed=21 + i, **kw) for i, s in enumerate(systems)]
    batch = B200MultiBatch(sims, **kw)
    batch.run()
    got = [sim.outcomes() for sim in sims]
    counts = {k: batch.last_counters[k] for k in COUNTS}
    batch.close()
    total = dict.fromkeys(COUNTS, 0)
    for sim, g in zip(sims, got):
        sim.run()
        for x, y in zip(g, sim.outcomes()):
            np.testing.assert_array_equal(x, y)
        for k in COUNTS:
            total[k] += sim.counters[k]
        sim.engine.close()
    assert counts == total


@pytest.mark.parametrize("precision,torque", [("mixed", "zero"), ("mixed", "centroid"), ("fp64", "zero")])
def test_batch_of_small_ligands_with_long_lists(precision, torque):
    """Two systems of at most 32 ligand atoms, more poses together than four for each of 16 warps per SM, and
    in FP64 enough for several poses a turn."""
    s = dataclasses.replace(system("c2"), r_start=12.0, r_escape=16.0)
    per = (3 if precision == "mixed" else 9) * 16 * _sms()
    _batch_equals_alone([s, dataclasses.replace(s, r_start=11.0)], per, 40, precision, torque)


@pytest.mark.parametrize("precision,torque", [("mixed", "centroid"), ("fp64", "zero")])
@pytest.mark.parametrize("n", [60, 300, 900])
def test_batch_of_large_ligands_with_short_lists(n, precision, torque):
    """Two systems of 176 ligand atoms: eight, four, two warps and one per pose in the ligand-atom kernel."""
    from pystarc_b200 import synth

    s = dataclasses.replace(synth.config3(scale=0.5, device="cuda"), r_start=20.0, r_escape=24.0)
    _batch_equals_alone([s, dataclasses.replace(s, r_start=19.0)], n, 40, precision, torque)


def test_contact_forces_in_a_batch():
    s = dataclasses.replace(system("c2"), r_start=12.0, r_escape=16.0)
    from pystarc_b200.multi import B200MultiBatch

    sims = [make_sim(s, 200, 60, "fp64", seed=3, use_lj=True), make_sim(system("c3"), 100, 60, "fp64", seed=4)]
    batch = B200MultiBatch(sims, steps_per_launch=8, launches_per_poll=2)
    batch.run()
    got = [sim.outcomes() for sim in sims]
    batch.close()
    for sim, g in zip(sims, got):
        sim.run()
        for x, y in zip(g, sim.outcomes()):
            np.testing.assert_array_equal(x, y)
        sim.engine.close()
