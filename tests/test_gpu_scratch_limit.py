"""A pool whose slots fit the device but whose split-step scratch does not runs the fused step, as it did when
that was the default; the next run that fits takes the split step again."""

import pytest

from tests.helpers import system
from tests.test_gpu_stepper import make_sim

pytestmark = pytest.mark.gpu

N = 20_000_000
SLOTS = N * (2 * 70 + 9)  # bytes: two slot buffers and the outcomes
SCRATCH = N * 113


def _group(sim):
    from pystarc_b200 import _lib

    g = _lib.C.c_int()
    sim.engine.handle.call("bd_get_launch", _lib.C.byref(g), None, None)
    return g.value


def test_pool_without_room_for_the_scratch():
    import torch

    s = system("c2")
    sim = make_sim(s, 64, 10)
    sim.run()  # kernels and the device system are loaded
    h = sim.engine.handle
    assert _group(sim) == 66
    big = make_sim(s, N, 1000, slots=N)
    big.engine.close()
    big.engine = sim.engine
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    room = SLOTS + SCRATCH // 2
    if free < room + (1 << 30):
        pytest.skip("device memory in use")
    filler = torch.empty(free - room, dtype=torch.uint8, device="cuda")
    try:
        big._setup()
        h.call("bd_sim_reset", None)
        h.call("bd_sim_run", 1, 2, None)
        c = big.read_counters()
        # trajectories may leave at the b-surface's return test, but nearly all take both steps
        assert 1.9 * N < c["steps"] <= 2 * N and c["started"] == N
        assert _group(big) == 65
    finally:
        del filler
        torch.cuda.empty_cache()
    sim.run()
    assert _group(sim) == 66
    sim.engine.close()
