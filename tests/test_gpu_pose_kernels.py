"""Force evaluation of pose batches: a block per pose (batches up to 24 poses per SM) and a warp per pose
(larger ones) sum the same terms in the same order, so a batch and its slices agree bit for bit, for poses
given as quaternions, as matrices and as lab-frame atoms; FP64 agrees with the 16-lane kernels to rounding."""

import numpy as np
import pytest

from tests.helpers import system
from tests.test_gpu_forces import make_engine, random_poses

pytestmark = pytest.mark.gpu

N = 3700  # above 24 poses on each of 148 SMs
SLICES = [(0, 1), (1, 38), (38, 700), (148, 3700)]


def _system(name):
    if name != "c3_half":
        return system(name)
    from pystarc_b200 import synth

    return synth.config3(scale=0.5, device="cuda")  # 176 ligand atoms: several rounds of a block


@pytest.mark.parametrize("sysname", ["c2", "c3", "c3_half"])
@pytest.mark.parametrize("precision,torque", [("fp64", "zero"), ("fp64", "centroid"), ("mixed", "centroid")])
def test_batches_and_their_slices_agree(sysname, precision, torque):
    from oracle.stepper import rotmats

    s = _system(sysname)
    eng = make_engine(s, precision, torque)
    body = s.lig_pos - s.lig_pos.mean(axis=0)
    eng.set_ligand(body, s.lig_q)
    c, q = random_poses(N, 4.0, 1.2 * s.r_start, 11)
    R = rotmats(q)
    pos = np.einsum("nij,kj->nki", R, body) + c[:, None, :]
    calls = [lambda a, b: eng.eval_poses(c[a:b], q[a:b]), lambda a, b: eng.eval_poses(c[a:b], R[a:b]),
             lambda a, b: eng(pos[a:b], s.lig_q, R[a:b], c[a:b])]
    whole = [f(0, N) for f in calls]
    for f, w in zip(calls, whole):
        for a, b in SLICES:
            for x, y in zip(f(a, b), w):
                np.testing.assert_array_equal(x, y[a:b])
    if precision == "fp64":
        eng.handle.call("bd_set_launch", 16, 128)
        ref = eng.eval_poses(c, q)
        for x, y in zip(whole[0], ref):
            # sums of at most a few thousand terms in another order: 1e-11 of the largest value
            np.testing.assert_allclose(x, y, rtol=0, atol=1e-11 * max(1.0, np.abs(y).max()))
    eng.close()
