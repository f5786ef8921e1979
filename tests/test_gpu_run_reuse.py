"""Runs that follow one another on one engine keep the device system, the buffers of equal size and the
captured graph where nothing they depend on changed; every run gives what a fresh engine gives."""

import numpy as np
import pytest

from tests.helpers import system
from tests.test_gpu_stepper import make_sim

pytestmark = pytest.mark.gpu


def _sim(s, eng, n, seed, cutoff, stats):
    from pystarc_b200.simulator import B200BatchSimulator

    mol1, mol2 = s.molecules()
    path = s.pathway_set()
    for p in path.reactions[0].criteria.pairs:
        p.distance_cutoff = cutoff
    return B200BatchSimulator(mol1, mol2, s.mobility(), path, s.params(n_traj=n, seed=seed, max_steps=80), eng,
                              termination="complete", steps_per_launch=16, launches_per_poll=2, stats=stats,
                              trace_capacity=0)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_runs_on_one_engine_equal_runs_on_fresh_engines(precision):
    s = system("c2")
    # (trajectories, seed, reaction cutoff, statistics): same again, other reactions, other size, statistics, back
    runs = [(300, 5, 4.5, False), (300, 5, 4.5, False), (300, 5, 9.0, False), (77, 5, 9.0, False),
            (300, 6, 4.5, True), (300, 5, 4.5, False)]
    shared = make_sim(s, 300, 80, precision).engine
    for n, seed, cutoff, stats in runs:
        got = _sim(s, shared, n, seed, cutoff, stats).run()
        fresh = make_sim(s, n, 80, precision).engine
        ref = _sim(s, fresh, n, seed, cutoff, stats).run()
        fresh.close()
        for k in ("outcome", "n_steps", "n_returns"):
            np.testing.assert_array_equal(got.sim_data[k], ref.sim_data[k])
        if stats:
            for k in ("min_dist", "radial_counts", "trans_matrix"):
                np.testing.assert_array_equal(got.sim_data[k], ref.sim_data[k])
        assert got.counters["steps"] == ref.counters["steps"]
    shared.close()


def test_reactions_changed_after_reset_are_refused_until_the_next_reset():
    from pystarc_b200 import _lib

    s = system("c2")
    sim = make_sim(s, 64, 80)
    h = sim.engine.handle
    sim._setup()
    h.call("bd_sim_reset", None)
    h.call("bd_set_reactions", 0, None, None, None, None, 1)
    with pytest.raises(_lib.BdError):
        h.call("bd_sim_run", 1, 4, None)
    h.call("bd_sim_reset", None)
    h.call("bd_sim_run", 1, 4, None)
    assert sim.read_counters()["reacted"] == 0
    sim.engine.close()
