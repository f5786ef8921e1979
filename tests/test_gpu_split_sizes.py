"""The split stepper at the sizes where its lists and pools can go wrong, against the fused stepper.

One slot, one more than a warp, one more than a block of the scalar kernel, sizes at which eight,
four and two warps share a pose of the sweep, and more slots than the force kernels have warps; launches of one step (begin and end without a middle kernel), of an
odd and of an even number of steps; pools with and without refill.  In FP64 and in mixed precision
both steppers sum every pose's terms in the same order, so outcomes are equal, not close.
"""

import numpy as np
import pytest

from tests.helpers import system
from tests.test_gpu_stepper import make_sim

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,slots,K", [(1, 1, 1), (33, 33, 3), (129, 129, 1), (400, 33, 2), (1500, 1500, 5), (3001, 3001, 4),
                                       (6001, 6001, 16)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("sysname", ["c2", "c3"])
def test_split_outcomes_equal_the_fused_steppers(n, slots, K, precision, sysname):
    s = system(sysname)
    outs = []
    for group in (65, 66):
        sim = make_sim(s, n, 60, precision, "centroid", slots=slots, steps_per_launch=K, launches_per_poll=4)
        sim.engine.handle.call("bd_set_launch", group, 128)
        res = sim.run()
        outs.append((sim.outcomes(), [res.counters[k] for k in ("steps", "reacted", "escaped", "returns", "overlap",
                                                                "bridge")]))
        sim.engine.close()
    for x, y in zip(outs[0][0], outs[1][0]):
        np.testing.assert_array_equal(x, y)
    assert outs[0][1] == outs[1][1]


@pytest.mark.parametrize("n,K", [(1, 1), (200, 3), (550, 2), (1100, 4), (2500, 2)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_large_ligands_shared_among_warps(n, K, precision):
    """A 176-atom ligand (ragged against 32 atoms a warp and a round): eight, four, two warps and one per pose."""
    from pystarc_b200 import synth

    s = synth.config3(scale=0.5, device="cuda")
    outs = []
    for group in (65, 66):
        sim = make_sim(s, n, 24, precision, "centroid", steps_per_launch=K, launches_per_poll=4, stats=True,
                       trace_capacity=0)
        sim.engine.handle.call("bd_set_launch", group, 128)
        res = sim.run()
        outs.append((sim.outcomes(), res.sim_data["min_dist"]))
        sim.engine.close()
    for x, y in zip(outs[0][0], outs[1][0]):
        np.testing.assert_array_equal(x, y)
    np.testing.assert_array_equal(outs[0][1], outs[1][1])
