"""What the engine's users have it do, as measurable cases.

Three kinds of work, each through the public entry points:

* ``forces`` -- net force, torque and energy of a batch of poses: ``B200ForceEngine.__call__`` with
  lab-frame atom positions (the reference engine's argument list) or ``eval_poses`` with centroids and
  quaternions (what training a surrogate and scoring poses use);
* ``run`` -- whole Brownian-dynamics runs: ``B200BatchSimulator.run()`` on a two-sphere,
  protein-ligand or protein-protein system, and ``B200MultiBatch.run()`` on several systems at once;
* ``mlp`` -- the surrogate network: ``MLPEnsemble.ensemble`` (inference of every member) and
  ``MLPEnsemble.grad`` (forward, loss and backward of one member on a batch).

The systems are the seeded synthetic ones of ``pystarc_b200.synth``, at full size or scaled down.  A
system (structures and grids) is built once per process; poses, noise seeds, weights and batches come
from the seed.
"""

from __future__ import annotations

import functools
import math
import types

import numpy as np
import torch

from pystarc_b200 import synth
from pystarc_b200.engine import B200ForceEngine
from pystarc_b200.multi import B200MultiBatch
from pystarc_b200.simulator import B200BatchSimulator
from pystarc_b200.surrogate import MLPEnsemble

DEV = "cuda:0"
EPS0 = 0.000142


def listed():
    return [
        # a script that steps or scores a few poses through the reference's own call: latency counts
        dict(name="call_few", kind="forces", system="ligand", scale=1.0, api="call", precision="fp64",
             torque="zero", poses=37),
        # exact targets for a surrogate's training set, mixed precision, one chunk of poses
        dict(name="poses_ligand_mixed", kind="forces", system="ligand", scale=1.0, api="poses", precision="mixed",
             torque="centroid", poses=100_000),
        # scoring protein-protein poses in full precision (1,401 x 1,701 atoms, bidirectional Born)
        dict(name="poses_protein_fp64", kind="forces", system="protein", scale=1.0, api="poses", precision="fp64",
             torque="centroid", poses=6_000),
        # two charged spheres to completion: validation against the analytic rate
        dict(name="run_spheres", kind="run", system="spheres", scale=1.0, precision="fp64", torque="zero",
             traj=100_000, max_steps=1_000_000, stats=False, hi="reference_gpu"),
        # the parameter file's default of 1,000 trajectories with the output files' statistics on
        dict(name="run_ligand_1k_stats", kind="run", system="ligand", scale=1.0, precision="fp64", torque="zero",
             traj=1_000, max_steps=1_024, stats=True, hi="reference_gpu"),
        # a first k_on estimate: some thousand trajectories followed into the contact region
        dict(name="run_ligand_8k", kind="run", system="ligand", scale=1.0, precision="mixed", torque="centroid",
             traj=8_000, max_steps=2_048, stats=False, hi="reference_gpu"),
        # production: as many trajectories as fit one pool, mixed precision
        dict(name="run_ligand_150k", kind="run", system="ligand", scale=1.0, precision="mixed", torque="zero",
             traj=150_000, max_steps=1_024, stats=False, hi="reference_gpu"),
        # the same in full precision, a ragged count
        dict(name="run_ligand_30k_fp64", kind="run", system="ligand", scale=1.0, precision="fp64", torque="zero",
             traj=30_011, max_steps=1_024, stats=False, hi="reference_gpu"),
        # protein-protein association with hydrodynamic interactions
        dict(name="run_protein_6k", kind="run", system="protein", scale=1.0, precision="mixed", torque="centroid",
             traj=6_000, max_steps=512, stats=False, hi="zuk"),
        # several receptor-ligand systems in one launch
        dict(name="run_batch", kind="run", system="batch", scale=1.0, precision="mixed", torque="zero",
             traj=4_000, max_steps=768, stats=False, hi="reference_gpu"),
        # surrogate inference on a step's trusted poses
        dict(name="mlp_ensemble", kind="mlp", op="ensemble", members=5, rows=100_000),
        # one training batch
        dict(name="mlp_grad", kind="mlp", op="grad", members=1, rows=8_192),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["forces", "run", "run", "run", "mlp"])
    if kind == "mlp":
        if rng.random() < 0.5:
            return dict(kind="mlp", op="ensemble", members=rng.randint(1, 8), rows=_log_int(rng, 1_000, 150_000))
        return dict(kind="mlp", op="grad", members=1, rows=32 * _log_int(rng, 8, 512))
    precision = rng.choice(["fp64", "mixed"])
    torque = rng.choice(["zero", "centroid"])
    if kind == "forces":
        system = rng.choice(["ligand", "protein"])
        top = 100_000 if system == "ligand" else 6_000
        return dict(kind="forces", system=system, scale=rng.choice([0.4, 0.7, 1.0]),
                    api=rng.choice(["call", "poses"]), precision=precision, torque=torque,
                    poses=_log_int(rng, 5, top))
    system = rng.choice(["spheres", "ligand", "ligand", "protein", "batch"])
    case = dict(kind="run", system=system, scale=rng.choice([0.4, 0.7, 1.0]), precision=precision, torque=torque,
                traj=0, max_steps=0, stats=False, hi="reference_gpu")
    if system == "spheres":
        case.update(scale=1.0, traj=_log_int(rng, 1_000, 100_000), max_steps=1_000_000)
    elif system == "ligand":
        case.update(traj=_log_int(rng, 100, 60_000), max_steps=rng.choice([512, 777, 1_024]))
        if case["traj"] <= 2_000:
            case["stats"] = rng.random() < 0.5
    elif system == "protein":
        case.update(traj=_log_int(rng, 100, 4_000), max_steps=rng.choice([128, 301, 512]),
                    hi=rng.choice(["reference_gpu", "zuk"]))
    else:
        case.update(scale=1.0, traj=_log_int(rng, 200, 4_000), max_steps=rng.choice([256, 512]))
    return case


# -------------------------------------------------------------------------------------------------
# systems
# -------------------------------------------------------------------------------------------------
ROWS = 103  # path rows of a trajectory: one every 10 steps, at most 1,024 steps with statistics on
BATCH_MEMBERS = (0, 3, 4, 15)  # members of the heterogeneous set of modest size


@functools.lru_cache(maxsize=None)
def _system(name, scale, index=0):
    if name == "spheres":
        return synth.config1()
    if name == "ligand":
        return synth.config2(scale=scale, device=DEV)
    if name == "protein":
        return synth.config3(scale=scale, device=DEV)
    return synth.config5(index, device=DEV)


def _engine(s, precision, torque):
    dip, quad, fpe = s.multipole_moments()
    moments = types.SimpleNamespace(dipole=dip, quadrupole=quad, four_pi_eps=fpe)
    return B200ForceEngine(**s.engine_kwargs(), multipole_expansion=moments, precision=precision, torque_mode=torque)


def _simulator(s, case, traj, seed):
    mol1, mol2 = s.molecules()
    p = s.params(n_traj=traj, seed=1 + seed, max_steps=case["max_steps"])
    if case["stats"]:
        p._output_cfg = types.SimpleNamespace(save_interval=10, full_paths=True, energetics=True)
    return B200BatchSimulator(mol1, mol2, s.mobility(), s.pathway_set(), p,
                              _engine(s, case["precision"], case["torque"]), hi_mode=case["hi"])


def _poses(s, n, seed):
    """Centroids from inside contact to beyond the b-sphere, uniform in distance, and random rotations."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    v = torch.randn(n, 3, generator=g, device=DEV, dtype=torch.float64)
    r_rec = float(np.linalg.norm(s.rec_pos, axis=1).max())
    r = 0.6 * r_rec + (1.1 * s.r_start - 0.6 * r_rec) * torch.rand(n, 1, generator=g, device=DEV, dtype=torch.float64)
    q = torch.randn(n, 4, generator=g, device=DEV, dtype=torch.float64)
    return v / v.norm(dim=1, keepdim=True) * r, q / q.norm(dim=1, keepdim=True)


def _rotations(q):
    w, x, y, z = q.unbind(1)
    return torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y),
                        2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x),
                        2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)], dim=1).reshape(-1, 3, 3)


def _ligand(s):
    return np.asarray(s.lig_pos) - np.asarray(s.lig_pos).mean(axis=0), np.asarray(s.lig_q)


# -------------------------------------------------------------------------------------------------
# surrogate network
# -------------------------------------------------------------------------------------------------
WIDTHS = (13, 256, 256, 256, 256, 6)


def _weights(members, seed):
    rng = np.random.default_rng(seed)
    return [np.concatenate([rng.uniform(-1, 1, n).astype(np.float32) / np.float32(math.sqrt(i))
                            for i, o in zip(WIDTHS[:-1], WIDTHS[1:]) for n in (i * o, o)]) for _ in range(members)]


def _features(rows, seed):
    """Pose features as the surrogate forms them: centroid, distance, quaternion and radial basis values."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    v = torch.randn(rows, 3, generator=g, device=DEV)
    r = 25 + 55 * torch.rand(rows, 1, generator=g, device=DEV)
    q = torch.randn(rows, 4, generator=g, device=DEV)
    q = q / q.norm(dim=1, keepdim=True)
    mu = torch.linspace(25, 80, 5, device=DEV)
    x = torch.cat([v / v.norm(dim=1, keepdim=True) * r / 80, r / 80, q * torch.sign(q[:, :1]),
                   torch.exp(-0.5 * ((r - mu) / 13.75) ** 2)], dim=1).contiguous()
    return x, torch.randn(rows, 6, generator=g, device=DEV)


# -------------------------------------------------------------------------------------------------
def prepare(case, seed):
    if case["kind"] == "mlp":
        ens = MLPEnsemble(n_members=case["members"], seed=seed)
        for m, w in enumerate(_weights(case["members"], seed)):
            ens.set_params(m, w)
        x, t = _features(case["rows"], seed)
        return dict(case=case, ens=ens, x=x, t=t)
    if case["kind"] == "forces":
        s = _system(case["system"], case["scale"])
        eng = _engine(s, case["precision"], case["torque"])
        body, q = _ligand(s)
        eng.set_ligand(body, q)
        c, quat = _poses(s, case["poses"], seed)
        R = _rotations(quat)
        state = dict(case=case, engine=eng, c=c, quat=quat, R=R, q=q)
        if case["api"] == "call":
            state["pos"] = torch.einsum("nij,aj->nai", R, torch.as_tensor(body, device=DEV)) + c[:, None, :]
        return state
    if case["system"] == "batch":
        sims = [_simulator(_system("batch", 1.0, k), case, case["traj"], seed + 100 * k) for k in BATCH_MEMBERS]
        return dict(case=case, batch=B200MultiBatch(sims))
    return dict(case=case, sim=_simulator(_system(case["system"], case["scale"]), case, case["traj"], seed))


def run(state):
    case = state["case"]
    if case["kind"] == "mlp":
        if case["op"] == "ensemble":
            mean, spread = state["ens"].ensemble(state["x"])
            return dict(mean=mean, spread=spread)
        loss, grad = state["ens"].grad(0, state["x"], state["t"])
        return dict(loss=loss, grad=grad)
    if case["kind"] == "forces":
        if case["api"] == "call":
            F, T, E = state["engine"](state["pos"], state["q"], state["R"], state["c"])
        else:
            F, T, E = state["engine"].eval_poses(state["c"], state["quat"])
        return dict(force=F, torque=T, energy=E)
    if case["system"] == "batch":
        return [_result(r) for r in state["batch"].run()]
    return _result(state["sim"].run())


def _result(r):
    d = {k: v for k, v in r.sim_data.items() if not isinstance(v, list) and not k.startswith(("encounter", "near_miss"))}
    n = r.n_trajectories
    if "path_steps" in r.sim_data:
        # rows per event become rows per trajectory, so that every run has the same layout
        sd = r.sim_data
        for name, width in (("path_steps", 6), ("energy_steps", 4)):
            full = np.zeros((n, ROWS, width))
            if sd[name]:
                rows = np.concatenate(sd[name])
                full[rows[:, 0].astype(np.int64), rows[:, 1].astype(np.int64) // 10] = rows[:, 2:]
            d[name] = full
        for kind in ("encounter", "near_miss"):
            for k in [k for k in sd if k.startswith(kind) and not k.endswith("traj")]:
                full = np.zeros((n,) + sd[k].shape[1:], sd[k].dtype)
                full[sd[kind + "_traj"]] = sd[k]
                d[k] = full
    d.update(n_reacted=r.n_reacted, n_escaped=r.n_escaped, n_max_steps=r.n_max_steps, total_steps=r.total_steps)
    return d


# -------------------------------------------------------------------------------------------------
# what a pass cannot do without
# -------------------------------------------------------------------------------------------------
STENCIL_FLOPS = 150  # trilinear value and gradient of one channel from 20 nodes
STEP_FLOPS = 800     # one trajectory's reaction test, dt, noise, move, rotation and bridge


def _grid_bytes(s):
    return sum(4 * np.asarray(g.data).size for g in s.elec_grids[:1] + s.born_grids[:1] + s.lig_born_grids[:1])


def _force_flops(s, near):
    """One pose: both channels at every ligand atom, and where it is near the receptor about an eighth of the
    receptor's atoms inside the ligand's Born grid."""
    rev = near * len(s.rec_q) / 8 if s.lig_born_grids else 0
    return STENCIL_FLOPS * (2 * len(s.lig_q) + rev)


def work(case):
    if case["kind"] == "mlp":
        mac = sum(i * o for i, o in zip(WIDTHS[:-1], WIDTHS[1:])) * case["rows"]
        n_par = sum(i * o + o for i, o in zip(WIDTHS[:-1], WIDTHS[1:]))
        if case["op"] == "ensemble":
            return dict(bytes=4 * (case["rows"] * (13 + 12) + n_par * case["members"]), flops=2 * mac * case["members"])
        return dict(bytes=4 * (case["rows"] * 19 + 2 * n_par), flops=6 * mac)
    if case["kind"] == "forces":
        s = _system(case["system"], case["scale"])
        pose_in = 8 * (3 * len(s.lig_q) + 12 if case["api"] == "call" else 7)
        # a pose reads its stencils' nodes; a large batch reads each grid once
        nodes = case["poses"] * 4 * 20 * (2 * len(s.lig_q) + len(s.rec_q) / 16)
        return dict(bytes=case["poses"] * (pose_in + 56) + min(nodes, _grid_bytes(s)),
                    flops=case["poses"] * _force_flops(s, 0.5))
    if case["system"] == "batch":
        parts = [_system("batch", 1.0, k) for k in BATCH_MEMBERS]
    else:
        parts = [_system(case["system"], case["scale"])]
    # two spheres: about 300 steps to an outcome; elsewhere most trajectories reach the step limit
    steps = case["traj"] * (300 if case["system"] == "spheres" else 0.7 * case["max_steps"])
    out = dict(bytes=0.0, flops=0.0)
    for s in parts:
        out["bytes"] += _grid_bytes(s) + case["traj"] * (9 + (250 if case["stats"] else 0))
        out["flops"] += steps * (STEP_FLOPS + _force_flops(s, 0.3))
    return out


# -------------------------------------------------------------------------------------------------
# the same in 64 bits, written out in torch
# -------------------------------------------------------------------------------------------------
class _Grid:
    def __init__(self, g):
        self.v = torch.as_tensor(np.asarray(g.data), device=DEV, dtype=torch.float64)
        self.o = torch.as_tensor(np.asarray(g.origin), device=DEV, dtype=torch.float64)
        self.h = torch.as_tensor(np.diag(np.asarray(g.delta)).copy(), device=DEV, dtype=torch.float64)
        self.n = torch.as_tensor(self.v.shape, device=DEV)

    def inside(self, x):
        """Strictly inside the box three spacings from every face."""
        return ((x > self.o + 3 * self.h) & (x < self.o + (self.n - 4) * self.h)).all(dim=-1)

    def value(self, x):
        u = (x - self.o) / self.h
        c = torch.floor(u)
        t = u - c
        c = c.long()
        out = 0.0
        for i in (0, 1):
            for j in (0, 1):
                for k in (0, 1):
                    w = ((t[:, 0] if i else 1 - t[:, 0]) * (t[:, 1] if j else 1 - t[:, 1])
                         * (t[:, 2] if k else 1 - t[:, 2]))
                    out = out + w * self.v[c[:, 0] + i, c[:, 1] + j, c[:, 2] + k]
        return out

    def value_and_gradient(self, x):
        """The trilinear interpolant, and its central difference over half a spacing per axis."""
        g = []
        for d in range(3):
            e = torch.zeros(3, device=DEV, dtype=torch.float64)
            e[d] = 0.5 * self.h[d]
            g.append((self.value(x + e) - self.value(x - e)) / self.h[d])
        return self.value(x), torch.stack(g, dim=1)


def _far_field(s, x, q):
    """Screened monopole, dipole and quadrupole of the receptor: radial force and energy, r at least 1 A."""
    dip, quad, fpe = (torch.as_tensor(v, device=DEV, dtype=torch.float64) for v in s.multipole_moments())
    lam = s.debye
    r = x.norm(dim=1).clamp(min=1.0)
    n = x / r[:, None]
    ex = torch.exp(-r / lam)
    V = float(np.sum(s.rec_q)) / (4 * math.pi * s.sdie * EPS0)
    p, w = n @ dip, ((n @ quad) * n).sum(dim=1)
    phi = V * ex / r + p / fpe * ex * (1 / r**2) * (1 + r / lam)
    phi = phi + w / fpe * ex / r**3 * (1 + r / lam + r**2 / (3 * lam**2))
    d = -V * ex * (1 / r**2 + 1 / (r * lam)) - p / fpe * ex * (2 / r**3 + 2 / (r**2 * lam) + 1 / (r * lam**2))
    d = d - w / fpe * ex * (3 / r**4 + 3 / (r**3 * lam) + 1 / (r**2 * lam**2) + 1 / (3 * r * lam**3))
    return -(q * d)[:, None] * n, q * phi


def _exact_forces(case, seed):
    s = _system(case["system"], case["scale"])
    c_all, quat = _poses(s, case["poses"], seed)
    R_all = _rotations(quat)
    body, lq = (torch.as_tensor(v, device=DEV, dtype=torch.float64) for v in _ligand(s))
    rec, rq = (torch.as_tensor(v, device=DEV, dtype=torch.float64) for v in (s.rec_pos, s.rec_q))
    elec, born, lborn = _Grid(s.elec_grids[0]), _Grid(s.born_grids[0]), _Grid(s.lig_born_grids[0])
    outs = []
    for i0 in range(0, len(c_all), 500):
        c, R = c_all[i0:i0 + 500], R_all[i0:i0 + 500]
        n = len(c)
        off = torch.einsum("nij,aj->nai", R, body)
        x = off + c[:, None, :]
        charged = (lq.abs() >= 1e-9).expand(n, -1)
        f = torch.zeros_like(x)
        e = torch.zeros(x.shape[:2], device=DEV, dtype=torch.float64)
        q = lq.expand(n, -1)
        m = elec.inside(x) & charged
        phi, g = elec.value_and_gradient(x[m])
        f[m] = -q[m][:, None] * g
        e[m] = q[m] * phi
        m = ~elec.inside(x) & charged
        f[m], e[m] = _far_field(s, x[m], q[m])
        m = born.inside(x) & charged
        phi, g = born.value_and_gradient(x[m])
        k = s.alpha * q[m] ** 2
        f[m] -= k[:, None] * g
        e[m] += k * phi
        F, T, E = f.sum(dim=1), torch.linalg.cross(off, f).sum(dim=1), e.sum(dim=1)
        # the ligand's Born grid at the receptor atoms, in the ligand frame: its force on the receptor, reversed
        y = torch.einsum("nji,nkj->nki", R, rec[None] - c[:, None, :])
        pose, atom = (lborn.inside(y) & (rq.abs() >= 1e-9)).nonzero(as_tuple=True)
        yy = y[pose, atom]
        _, g = lborn.value_and_gradient(yy)
        g = -s.alpha * (rq[atom] ** 2)[:, None] * g
        fr = torch.zeros(n, 3, device=DEV, dtype=torch.float64).index_add_(0, pose, g)
        tr = torch.zeros(n, 3, device=DEV, dtype=torch.float64).index_add_(0, pose, torch.linalg.cross(yy, g))
        F = F - torch.einsum("nij,nj->ni", R, fr)
        T = T - torch.einsum("nij,nj->ni", R, tr)
        outs.append((F, T if case["torque"] == "centroid" else torch.zeros_like(T), E))
    F, T, E = (torch.cat(v) for v in zip(*outs))
    return dict(force=F, torque=T, energy=E)


def _exact_mlp(case, seed):
    x, t = (v.double() for v in _features(case["rows"], seed))
    outs = []
    for w in _weights(case["members"], seed):
        p = torch.as_tensor(w, device=DEV).double().requires_grad_(case["op"] == "grad")
        a, at = x, 0
        for layer, (i, o) in enumerate(zip(WIDTHS[:-1], WIDTHS[1:])):
            a = a @ p[at:at + i * o].reshape(o, i).T + p[at + i * o:at + i * o + o]
            at += i * o + o
            if layer + 2 < len(WIDTHS):
                a = torch.nn.functional.silu(a)
        if case["op"] == "grad":
            loss = ((a - t) ** 2).mean()
            loss.backward()
            return dict(loss=float(loss.detach()), grad=p.grad)
        outs.append(a)
    y = torch.stack(outs)
    mean = y.mean(dim=0)
    return dict(mean=mean, spread=((y - mean) ** 2).mean(dim=0).sqrt())


def exact(case, seed):
    if case["kind"] == "mlp":
        return _exact_mlp(case, seed)
    if case["kind"] == "forces":
        return _exact_forces(case, seed)
    return None  # outcomes and step counts are whole numbers of one noise stream
