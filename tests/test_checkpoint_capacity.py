"""A checkpoint whose pool has another capacity than this run's default pool is resumed.

The default capacity follows from how many trajectories of the stepper's kernel are resident, so it changes
with the kernels; the checkpoint says what its pool was, and the resumed run takes a pool of that size.
A run that asks for a pool size of its own still refuses a checkpoint of another.  Device calls are
answered by the mocked handle of the multi-rank tests.
"""

import numpy as np
import pytest

from tests.helpers import system
from tests.test_multi_rank import _FakeEngine, _FakeHandle

N = 64
LIVE = 10


class _Handle(_FakeHandle):
    def __init__(self, s, default):
        super().__init__(s)
        self.default, self.cap, self.restored = default, 0, None

    def call(self, name, *args):
        if name == "bd_sim_configure":
            sp = args[0]._obj
            self.cap = min(int(sp.slots) or self.default, int(sp.n_traj))
        elif name == "bd_sim_capacity":
            args[0]._obj.value = self.cap
        elif name == "bd_sim_snapshot":
            for width, a in zip((3, 4, 1, 1, 1, 1), args[:6]):
                for i in range(width):
                    for slot in range(LIVE):
                        a[i * self.cap + slot] = 10 * slot + i
            args[6]._obj.value = LIVE
            return 0
        elif name == "bd_sim_restore":
            live = int(args[6])
            self.restored = [[[a[i * self.cap + slot] for slot in range(live)] for i in range(width)]
                             for width, a in zip((3, 4, 1, 1, 1, 1), args[:6])]
            return 0
        return super().call(name, *args)


def _sim(default, tmp_path, slots=0, interval=0):
    from pystarc_b200.simulator import B200BatchSimulator

    s = system("two_sphere")
    mol1, mol2 = s.molecules()
    p = s.params(n_traj=N, max_steps=20)
    p._work_dir = str(tmp_path)
    p.checkpoint_interval = interval
    eng = _FakeEngine(s)
    eng.handle = _Handle(s, default)
    sim = B200BatchSimulator(mol1, mol2, s.mobility(), s.pathway_set(), p, eng, termination="complete", slots=slots)
    return sim


def _saved(default, tmp_path):
    sim = _sim(default, tmp_path)
    sim._setup()
    sim.engine.handle.call("bd_sim_reset", None)
    return sim.save_checkpoint(tmp_path / "checkpoint_b200.npz")


@pytest.mark.parametrize("saved,now", [(16, 32), (32, 16), (16, 1000), (1000, 16)])
def test_a_pool_of_another_capacity_is_resumed(saved, now, tmp_path, capsys):
    path = _saved(saved, tmp_path)
    sim = _sim(now, tmp_path)
    sim._setup()
    sim.load_checkpoint(path)
    assert sim.engine.handle.cap == min(saved, N)
    assert sim.engine.handle.restored == [[[float(10 * slot + i) for slot in range(LIVE)] for i in range(width)]
                                          for width in (3, 4, 1, 1, 1, 1)]
    sim = _sim(now, tmp_path, interval=1)  # a whole run finds the file and goes on from it
    sim.run()
    assert "Starting fresh" not in capsys.readouterr().out
    assert sim.engine.handle.restored is not None


def test_a_pool_size_that_was_asked_for_is_kept(tmp_path):
    path = _saved(16, tmp_path)
    sim = _sim(16, tmp_path, slots=24)
    sim._setup()
    with pytest.raises(ValueError, match="slot capacity 16 != 24"):
        sim.load_checkpoint(path)
    assert sim.engine.handle.cap == 24 and sim.engine.handle.restored is None


@pytest.mark.parametrize("cap", [0, -1, N + 1])
def test_a_capacity_that_no_run_can_have_is_refused(cap, tmp_path):
    path = _saved(16, tmp_path)
    d = dict(np.load(path))
    np.savez(path, **{**d, "cap": cap})
    sim = _sim(32, tmp_path)
    sim._setup()
    with pytest.raises(ValueError, match="slot capacity"):
        sim.load_checkpoint(path)
    assert sim.engine.handle.cap == 32


@pytest.mark.gpu
def test_resumed_on_the_device(tmp_path):
    """200 trajectories from a pool of 64, resumed by a run whose default pool holds all of them."""
    from tests.test_gpu_stepper import make_sim

    s = system("c2")
    whole = make_sim(s, 200, 300, steps_per_launch=8)
    whole.run()
    first = make_sim(s, 200, 300, steps_per_launch=8, slots=64)
    first.run(max_launches=16)
    path = first.save_checkpoint(tmp_path / "c.npz")
    rest = make_sim(s, 200, 300, steps_per_launch=8)
    rest._setup()
    rest.engine.handle.call("bd_sim_reset", None)
    rest.load_checkpoint(path)
    h = rest.engine.handle
    for _ in range(200):
        h.call("bd_sim_run", 4, 8, None)
        c = rest.read_counters()
        if c["reacted"] + c["escaped"] + c["max_steps"] == 200:
            break
    for x, y in zip(whole.outcomes(), rest.outcomes()):
        np.testing.assert_array_equal(x, y)
    for sim in (whole, first, rest):
        sim.engine.close()
