"""The first launch of a pool goes to the stream as it is and the graphs are built behind it: however the
launches of a run are grouped into calls, and on whichever stream, every trajectory takes the same steps."""

import numpy as np
import pytest

from tests.helpers import system
from tests.test_gpu_stepper import make_sim

pytestmark = pytest.mark.gpu


def _snapshot(sim, n):
    from pystarc_b200 import _lib

    c, q = np.zeros(3 * n), np.zeros(4 * n)
    traj, nstep, rets = (np.zeros(n, dtype=np.int32) for _ in range(3))
    status, live, ctr = np.zeros(n, dtype=np.int8), _lib.C.c_int32(), np.zeros(_lib.N_CTR, dtype=np.uint64)
    i32 = _lib.C.c_int32
    sim.engine.handle.call("bd_sim_snapshot", _lib.ptr(c), _lib.ptr(q), _lib.ptr(traj, i32), _lib.ptr(nstep, i32),
                           _lib.ptr(rets, i32), _lib.ptr(status, _lib.C.c_int8), _lib.C.byref(live),
                           _lib.ptr(ctr, _lib.C.c_uint64))
    m = live.value
    order = np.argsort(traj[:m])
    return np.concatenate([c.reshape(3, n)[:, :m], q.reshape(4, n)[:, :m], nstep[None, :m]])[:, order]


# (launches, steps) of each call: 18 steps in all
CALLS = [[(6, 3)], [(1, 3)] * 6, [(2, 3), (4, 3)], [(3, 3), (9, 1)], [(0, 3), (6, 3)], [(1, 18)]]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("side_stream", [False, True])
def test_calls_of_any_grouping_take_the_same_steps(precision, side_stream):
    import torch

    s, n = system("c2"), 300
    stream = torch.cuda.Stream().cuda_stream if side_stream else None
    rows = []
    for group, calls in [(65, CALLS[0])] + [(66, c) for c in CALLS]:
        sim = make_sim(s, n, 1_000_000, precision, "centroid")
        h = sim.engine.handle
        h.call("bd_set_launch", group, 128)
        for _ in range(2):  # a second run on the engine keeps the graphs of the first
            sim._setup()
            h.call("bd_sim_reset", None)
            torch.cuda.synchronize()
            for launches, steps in calls:
                h.call("bd_sim_run", launches, steps, stream)
            torch.cuda.synchronize()
            rows.append(_snapshot(sim, n))
        sim.engine.close()
    for r in rows[1:]:
        np.testing.assert_array_equal(r, rows[0])


@pytest.mark.parametrize("launches_per_poll", [1, 2, 5])
def test_batches_of_any_grouping_take_the_same_steps(launches_per_poll):
    from pystarc_b200.multi import B200MultiBatch

    sims = [make_sim(system(name), 150, 60, seed=3 + i) for i, name in enumerate(("c2", "two_sphere", "c3"))]
    batch = B200MultiBatch(sims, steps_per_launch=8, launches_per_poll=launches_per_poll)
    batch.run()
    got = [sim.outcomes() for sim in sims]
    batch.close()
    for sim, g in zip(sims, got):
        sim.run()
        for x, y in zip(g, sim.outcomes()):
            np.testing.assert_array_equal(x, y)
        sim.engine.close()
