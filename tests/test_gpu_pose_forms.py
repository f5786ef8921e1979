"""Batches of poses take one kernel, a block per pose or a warp per pose by their size and by the work of a
pose.  Every form sums the same terms in the same order, so a batch and its slices agree bit for bit: with
contact forces, for each choice of force terms, and for systems on either side of every line."""

import dataclasses

import numpy as np
import pytest

from tests.helpers import system
from tests.test_gpu_forces import make_engine, random_poses

pytestmark = pytest.mark.gpu

# poses per SM on either side of the lines at 6, 9, 12, 20 and 24
EDGES = (1, 6, 6.1, 9, 9.1, 12, 12.1, 20, 20.1, 24, 24.1)


def _systems(name):
    from pystarc_b200 import synth

    if name == "c2_full":  # 3,201 receptor atoms: 101 units of work
        return synth.config2(device="cuda")
    if name == "c3_half":  # 213 + 176 atoms: 13 units, and 6 without the sweep
        return synth.config3(scale=0.5, device="cuda")
    if name == "c3_half_no_sweep":
        return dataclasses.replace(synth.config3(scale=0.5, device="cuda"), lig_born_grids=[])
    if name == "c3_no_sweep":  # 1,401 ligand atoms: 44 units
        return dataclasses.replace(synth.config3(device="cuda"), lig_born_grids=[])
    return system(name)


@pytest.mark.parametrize("sysname", ["c2", "c2_full", "c3_half", "c3_half_no_sweep", "c3_no_sweep"])
@pytest.mark.parametrize("precision,torque", [("fp64", "centroid"), ("mixed", "zero"), ("mixed", "centroid")])
@pytest.mark.parametrize("contact", [False, True])
def test_every_form_gives_the_same_bits(sysname, precision, torque, contact):
    import torch

    from oracle.stepper import rotmats
    from pystarc_b200 import _lib

    s = _systems(sysname)
    eng = make_engine(s, precision, torque, use_lj=contact)
    body = s.lig_pos - s.lig_pos.mean(axis=0)
    eng.set_ligand(body, s.lig_q)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = int(26 * sms)
    c, q = random_poses(n, 4.0, 1.2 * s.r_start, 12)
    R = rotmats(q)
    few = int(7 * sms)
    pos = np.einsum("nij,kj->nki", R[:few], body) + c[:few, None, :]
    whole = eng.eval_poses(c, q)
    assert np.abs(whole[0]).max() > 0
    for per_sm in EDGES:
        m = int(per_sm * sms)
        for x, y in zip(eng.eval_poses(c[n - m:], q[n - m:]), whole):
            np.testing.assert_array_equal(x, y[n - m:])
    for m in (3, few):  # lab-frame atoms against one another: the placed atoms differ in the last bit
        for x, y in zip(eng(pos[:m], s.lig_q, R[:m], c[:m]), eng(pos, s.lig_q, R[:few], c[:few])):
            np.testing.assert_array_equal(x, y[:m])
    for terms in (_lib.TERM_GRID, _lib.TERM_FARFIELD | _lib.TERM_REV_BORN, 8):
        part = eng.eval_poses(c, q, terms=terms)
        for m in (2, few):
            for x, y in zip(eng.eval_poses(c[:m], q[:m], terms=terms), part):
                np.testing.assert_array_equal(x, y[:m])
    eng.close()
