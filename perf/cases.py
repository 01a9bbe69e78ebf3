"""The work that users of this framework have it do, as cases to time.

Every case goes through the public entry points.  The chains are runs of
consecutive residues of the committed 4 x 1,000-residue chain
(workloads/c5_multidomain_4x1000res.npz: all atoms, folded-protein density),
so sizes range from a peptide to the whole 65,294 atoms.  A case's seed gives
the coordinates: a rigid turn of the chain and a thermal jitter of 0.02 A per
atom, and the seed of the sampler.

kinds
  score     one energy of a particle list (PhysicsEngine.energy_terms): what
            a script or the GUI asks for between edits
  rescore   new frames of one chain loaded into a resident batch and scored
            (DeviceBatch.load_coords + energy_terms): a trajectory's energies
  forces    energy and gradient of one chain: evaluate() eagerly, as one
            replayed CUDA graph, or through autograd (EnergyModel)
  ensemble  PhysicsEngine.generate_ensemble, particle lists in and out: one
            candidate on an engine that the program keeps, several as the
            first call of a script (an engine of its own)
  landscape PhysicsEngine.run_landscape_segment: snapshots and their energies
  batch     BatchedEnsemble.run: many different chains, host coordinates in
            and out, 280-400 K
  mala      gradient-guided torsion sampling (MALARunner.run)
  replica   one interval of replica exchange (MALA : torsion moves 1 : 3)
  contacts  distance and contact matrices of an ensemble on the device
"""
import functools
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "protein-structure-analysis_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from protein_physics_b200 import BondTopology, Particle, PhysicsEngine, flatten  # noqa: E402
from protein_physics_b200.analysis import compute_contact_freq_matrix, compute_mean_dist_matrix  # noqa: E402
from protein_physics_b200.autograd import EnergyModel  # noqa: E402
from protein_physics_b200.device import DeviceBatch  # noqa: E402
from protein_physics_b200.mc import K_BOLTZMANN, BatchedEnsemble  # noqa: E402
from protein_physics_b200.replica import ReplicaExchange, geometric_ladder  # noqa: E402
from protein_physics_b200.torsion import MALARunner  # noqa: E402

RESIDUES = 4030        # of the source chain
ATOMS_PER_RESIDUE = 16.2


def listed():
    return [
        # one energy of a short chain: latency, launches and host work
        {"name": "score_64res", "kind": "score", "residues": 64, "precision": "mixed"},
        # 48 frames of a 300-residue trajectory
        {"name": "rescore_48x300res", "kind": "rescore", "residues": 300, "frames": 48, "precision": "mixed"},
        # gradient steps of a small chain in full precision
        {"name": "forces_150res_fp64", "kind": "forces", "residues": 150, "precision": "fp64", "api": "evaluate"},
        # a differentiable loss on a 1,000-residue chain (forward and backward)
        {"name": "forces_1000res_autograd", "kind": "forces", "residues": 1000, "precision": "mixed",
         "api": "autograd"},
        # the largest single chain, replayed as one graph
        {"name": "forces_4030res_graph", "kind": "forces", "residues": 4030, "precision": "mixed", "api": "graph"},
        # one candidate of a 300-residue chain at 300 K
        {"name": "ensemble_300res", "kind": "ensemble", "residues": 300, "candidates": 1, "steps": 400},
        # a few candidates of a short chain
        {"name": "ensemble_16x64res", "kind": "ensemble", "residues": 64, "candidates": 16, "steps": 200},
        # a landscape segment: snapshots with their energies
        {"name": "landscape_200res", "kind": "landscape", "residues": 200, "snapshots": 5, "steps": 60},
        # production sampling: 256 chains of 50-600 residues, 50 proposals each
        {"name": "batch_256", "kind": "batch", "chains": 256, "smallest": 50, "largest": 600, "steps": 50},
        # all-bond Langevin proposals of a 1,000-residue chain
        {"name": "mala_1000res", "kind": "mala", "residues": 1000, "proposals": 24},
        # one interval of 8 replicas of a 600-residue chain, 300-450 K
        {"name": "replica_8x600res", "kind": "replica", "residues": 600, "replicas": 8, "sweeps": 24},
        # contact analysis of 1,000 snapshots of a 601-residue chain
        {"name": "contacts_601x1000", "kind": "contacts", "residues": 601, "snapshots": 1000},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["score", "rescore", "forces", "forces", "ensemble", "ensemble", "landscape", "batch", "batch",
                       "mala", "replica", "contacts"])
    if kind == "score":
        return {"kind": kind, "residues": _log_int(rng, 20, 1000), "precision": rng.choice(["mixed", "fp64"])}
    if kind == "rescore":
        return {"kind": kind, "residues": _log_int(rng, 40, 600), "frames": _log_int(rng, 2, 64),
                "precision": rng.choice(["mixed", "mixed", "fp64"])}
    if kind == "forces":
        return {"kind": kind, "residues": _log_int(rng, 20, 4030), "precision": rng.choice(["mixed", "mixed", "fp64"]),
                "api": rng.choice(["evaluate", "autograd", "graph"])}
    if kind == "ensemble":
        return {"kind": kind, "residues": _log_int(rng, 30, 500), "candidates": _log_int(rng, 1, 24),
                "steps": _log_int(rng, 50, 300)}
    if kind == "landscape":
        return {"kind": kind, "residues": _log_int(rng, 30, 400), "snapshots": rng.randint(2, 6),
                "steps": _log_int(rng, 20, 100)}
    if kind == "batch":
        a = _log_int(rng, 30, 200)
        return {"kind": kind, "chains": _log_int(rng, 8, 256), "smallest": a, "largest": a + rng.randint(20, 300),
                "steps": _log_int(rng, 10, 50)}
    if kind == "mala":
        return {"kind": kind, "residues": _log_int(rng, 50, 2000), "proposals": rng.randint(8, 32)}
    if kind == "replica":
        return {"kind": kind, "residues": _log_int(rng, 60, 600), "replicas": rng.randint(2, 8),
                "sweeps": 4 * rng.randint(2, 6)}
    return {"kind": "contacts", "residues": _log_int(rng, 30, 1500), "snapshots": _log_int(rng, 20, 1000)}


# ---- inputs ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=1)
def _source():
    d = np.load(os.path.join(_ROOT, "workloads", "c5_multidomain_4x1000res.npz"), allow_pickle=False)
    return {k: d[k] for k in d.files}


@functools.lru_cache(maxsize=256)
def _chain(residues, which=0, sidechain_pairs=False):
    """(xyz, charge, radius, epsilon, topology) of `residues` residues of
    the source chain; which moves the window along it; sidechain_pairs: with
    the landscape sampler's concerted moves."""
    d = _source()
    ridx = d["res_idx"]
    r0 = (411 + 619 * which) % max(1, RESIDUES - residues + 1) if residues < RESIDUES else 0
    a, b = np.searchsorted(ridx, [r0, r0 + residues])
    topo = BondTopology()
    topo.build([str(v) for v in d["resnames"][a:b]], [str(v) for v in d["atomnames"][a:b]],
               [int(v) - r0 for v in ridx[a:b]])
    if sidechain_pairs:
        topo.identify_concerted_sidechain_pairs(d["xyz"][a:b].astype(np.float64))
    return (d["xyz"][a:b].astype(np.float64), d["charge"][a:b].astype(np.float64),
            d["radius"][a:b].astype(np.float64), d["epsilon"][a:b].astype(np.float64), topo)


def _coords(xyz, rng):
    """A rigid turn about the chain's centre and a thermal jitter."""
    q = rng.normal(size=4)
    w, x, y, z = q / np.linalg.norm(q)
    R = np.array([[1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w)],
                  [2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w)],
                  [2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)]])
    return np.ascontiguousarray((xyz - xyz.mean(0)) @ R.T + 0.02 * rng.normal(size=xyz.shape))


def _particles(x, q, r, e):
    return [Particle(*p, c, s, t) for p, c, s, t in zip(x.tolist(), q.tolist(), r.tolist(), e.tolist())]


def _batch_chains(case, rng):
    """Chains of a batch: sizes spread evenly over the range, several copies
    (with coordinates of their own) of each of up to 24 different chains."""
    n = case["chains"]
    kinds = max(1, min(24, n))
    sizes = [int(round(case["smallest"] + (case["largest"] - case["smallest"]) * k / max(1, kinds - 1)))
             for k in range(kinds)]
    out = []
    for k in range(n):
        xyz, q, r, e, topo = _chain(sizes[k % kinds], k % kinds)
        out.append((_coords(xyz, rng), q, r, e, flatten(topo)))
    return out


def prepare(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    state = {"case": case}
    if kind == "contacts":
        n, s = case["residues"], case["snapshots"]
        # a compact self-avoiding-like backbone (3.8 A steps, drifting) with per-snapshot fluctuations
        step = rng.normal(size=(n, 3))
        step = 3.8 * step / np.linalg.norm(step, axis=1, keepdims=True)
        base = torch.as_tensor(np.cumsum(step, 0), device="cuda")
        g = torch.Generator(device="cuda").manual_seed(int(seed))
        state["coords"] = base + 1.5 * torch.randn((s, n, 3), generator=g, dtype=torch.float64, device="cuda")
        return state
    if kind == "batch":
        chains = _batch_chains(case, rng)
        n = case["chains"]
        temps = geometric_ladder(280.0, 400.0, n) * K_BOLTZMANN
        ens = BatchedEnsemble(chains, temps, seed=seed)
        start = torch.empty((ens.batch.natoms, 3), dtype=torch.float64, pin_memory=True)
        start.copy_(torch.from_numpy(np.concatenate([c[0] for c in chains])))
        state.update(ens=ens, start=start)
        return state
    xyz, q, r, e, topo = _chain(case["residues"], sidechain_pairs=kind == "landscape")
    x = _coords(xyz, rng)
    if kind == "score":
        state.update(engine=PhysicsEngine(precision=case["precision"]), particles=_particles(x, q, r, e), topo=topo)
    elif kind in ("ensemble", "landscape"):
        state.update(seed=seed, engine=PhysicsEngine(seed=seed), particles=_particles(x, q, r, e), topo=topo)
    elif kind == "rescore":
        flat = flatten(topo)
        state["batch"] = DeviceBatch([(x, q, r, e, flat)] * case["frames"], precision=case["precision"])
        state["frames"] = torch.as_tensor(_frames(x, case["frames"], rng).reshape(-1, 3), device="cuda")
    elif kind == "forces":
        system = (x, q, r, e, flatten(topo))
        if case["api"] == "autograd":
            state["model"] = EnergyModel([system], precision=case["precision"])
            state["x"] = torch.as_tensor(x, device="cuda").requires_grad_()
        else:
            state["batch"] = DeviceBatch([system], precision=case["precision"])
    elif kind == "mala":
        batch = DeviceBatch([(x, q, r, e, flatten(topo))])
        state.update(batch=batch, runner=MALARunner(batch, 300.0 * K_BOLTZMANN, seed))
    else:
        state["rex"] = ReplicaExchange((x, q, r, e, flatten(topo)), geometric_ladder(300.0, 450.0, case["replicas"]),
                                       seed)
    return state


def _frames(x, frames, rng):
    return x + 0.02 * rng.normal(size=(frames, *x.shape))


# ---- one pass -------------------------------------------------------------------------
def _positions(members):
    return [np.array([(p.x, p.y, p.z) for p in m]) for m in members]


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "score":
        return state["engine"].energy_terms(state["particles"], state["topo"])
    if kind == "rescore":
        state["batch"].load_coords(state["frames"])
        return state["batch"].energy_terms()
    if kind == "forces":
        if case["api"] == "autograd":
            x = state["x"]
            x.grad = None
            E = state["model"](x)
            E.sum().backward()
            return {"energy": E.detach(), "grad": x.grad}
        terms, grad = state["batch"].evaluate(graph=case["api"] == "graph")
        return {"terms": terms, "grad": grad}
    if kind == "ensemble":
        engine = state["engine"] if case["candidates"] == 1 else PhysicsEngine(seed=state["seed"])
        return _positions(engine.generate_ensemble(state["particles"], state["topo"], case["candidates"],
                                                   case["steps"], 300.0 * K_BOLTZMANN))
    if kind == "landscape":
        snaps, energies, cur_max = state["engine"].run_landscape_segment(
            state["particles"], state["topo"], case["snapshots"], case["steps"], 300.0 * K_BOLTZMANN)
        return {"snapshots": _positions(snaps), "energies": energies, "cur_max": cur_max}
    if kind == "batch":
        xyz = state["ens"].run(case["steps"], xyz=state["start"])
        st = state["ens"].state()
        return {"xyz": xyz, "energy": st["energy"], "accepted": st["n_accepted"], "steps": st["step"]}
    if kind == "mala":
        st = state["runner"].run(case["proposals"], graph=True)
        return {"xyz": state["batch"].xyz, "energy": st["energy"], "accepted": st["n_accepted"],
                "gradient": state["runner"].cur.g}
    if kind == "replica":
        rex = state["rex"]
        rex.interval(case["sweeps"])
        return {"xyz": rex.batch.xyz, "terms": rex.terms, "sys_of_temp": rex.sys_of_temp, "accepts": rex.accepts}
    return {"mean": compute_mean_dist_matrix(state["coords"]),
            "contacts": compute_contact_freq_matrix(state["coords"], 8.0)}


# ---- the work a pass cannot do without ---------------------------------------------------
# Operations per term: pair 47 (backward 104), HCT 21 (derivative 25), a
# neighbour's SASA step 11.  A pair within 12 A is one pair term, one within
# 14 A two HCT terms (both directions).
def _neighbours(residues):
    """Atoms within 14 A of an atom (measured on windows of the source chain:
    235 at 64 residues, 320 at 300, 520 at 1,000, 602 at 4,000)."""
    return min(600.0, 235.0 + 0.29 * max(0, residues - 64))


def _energy_flops(residues):
    nb = _neighbours(residues)
    return ATOMS_PER_RESIDUE * residues * nb / 2 * (0.70 * 47 + 2 * 21 + 0.2 * 11)


def _force_flops(residues):
    nb = _neighbours(residues)
    return ATOMS_PER_RESIDUE * residues * nb / 2 * (0.70 * 104 + 2 * 25 + 0.2 * 22)


def _proposal_flops(residues):
    """One proposal under generate_ensemble's policy: per atom of the chain 66
    pair terms (old and new), 68 HCT terms and 39 SASA steps at 719 neighbours
    (counted on the 300-residue compact chain)."""
    return ATOMS_PER_RESIDUE * residues * _neighbours(residues) / 719 * (66 * 47 + 68 * 21 + 39 * 11)


def work(case):
    kind = case["kind"]
    if kind == "contacts":
        n, s = case["residues"], case["snapshots"]
        return {"bytes": 2 * (24.0 * n * s + 8.0 * n * n), "flops": 2 * 10.0 * s * n * (n - 1) / 2}
    if kind == "batch":
        mean = (case["smallest"] + case["largest"]) / 2
        atoms = ATOMS_PER_RESIDUE * mean * case["chains"]
        return {"bytes": 48.0 * atoms + 24.0 * atoms,
                "flops": case["chains"] * (_energy_flops(mean) + case["steps"] * _proposal_flops(mean))}
    n, res = ATOMS_PER_RESIDUE * case["residues"], case["residues"]
    atom_in = 24.0 + 24.0  # coordinates and parameters
    if kind == "score":
        return {"bytes": atom_in * n, "flops": _energy_flops(res)}
    if kind == "rescore":
        return {"bytes": (24.0 * case["frames"] + 24.0) * n, "flops": case["frames"] * _energy_flops(res)}
    if kind == "forces":
        return {"bytes": (atom_in + 24.0) * n, "flops": _energy_flops(res) + _force_flops(res)}
    if kind == "ensemble":
        c = case["candidates"]
        return {"bytes": (atom_in + 24.0 * c) * n, "flops": c * (_energy_flops(res) + case["steps"] * _proposal_flops(res))}
    if kind == "landscape":
        k = case["snapshots"]
        return {"bytes": (atom_in + 24.0 * k) * n,
                "flops": _energy_flops(res) * (k + 1) + k * case["steps"] * _proposal_flops(res)}
    if kind == "mala":
        return {"bytes": (atom_in + 24.0) * n,
                "flops": case["proposals"] * (_energy_flops(res) + _force_flops(res))}
    rep, sw = case["replicas"], case["sweeps"]
    n_mala = round(sw / 4)
    return {"bytes": rep * 72.0 * n,
            "flops": rep * ((n_mala + 1) * (_energy_flops(res) + _force_flops(res)) + (sw - n_mala) * _proposal_flops(res)
                            + 2 * _energy_flops(res))}


# ---- 64-bit values ----------------------------------------------------------------------
# The reference energy in plain torch, FP64 (constants of physics_engine.cpp
# :181-196): HCT Born radii over pairs within 14 A, Debye-Hueckel + GB + LJ +
# capped hard core over non-excluded pairs within 12 A, the order-dependent
# SASA recurrence over the cell-scan order, dihedral and disulfide terms.
def _hct(r, r2, ri, rj):
    L, U = torch.maximum((r - rj).abs(), ri), r + rj
    v = 1 / L - 1 / U + (r2 - rj * rj + ri * ri) / (4 * r2 * ri * ri) * torch.log(L / U)
    return torch.where(ri >= U, torch.zeros_like(v), v)


def _pairs_within(x, cut2):
    """(I, J), I < J, with r^2 < cut2, by blocks of rows."""
    n, I, J = len(x), [], []
    for a in range(0, n, 2048):
        d = x[a:a + 2048, None, :] - x[None, a:, :]
        i, j = torch.nonzero((d * d).sum(2) < cut2, as_tuple=True)
        keep = j > i
        I.append(i[keep] + a)
        J.append(j[keep] + a)
    return torch.cat(I), torch.cat(J)


def _exact_energy(x, q, r, e, flat):
    """[sasa, dihedral, disulfide, pairs, total] as a function of x [n, 3]."""
    dev, n = x.device, len(x)
    as_t = lambda v, t=torch.float64: torch.tensor(np.asarray(v), dtype=t, device=dev)  # noqa: E731
    q, r, e = as_t(q), as_t(r), as_t(e)
    with torch.no_grad():
        I, J = _pairs_within(x, 196.0)
        lo = x.min(0).values - (14.0 + 1e-6)
        hi = x.max(0).values
        cs = 14.0 + 1e-6
        dims = torch.clamp(torch.ceil((hi - lo + 2 * cs) / cs).long(), min=1)
        c = torch.floor((x - lo) / cs).long()
        key = c[:, 0] + dims[0] * (c[:, 1] + dims[1] * c[:, 2])
        rank = torch.empty(n, dtype=torch.long, device=dev)
        rank[torch.argsort(key, stable=True)] = torch.arange(n, device=dev)  # the scan order of a row
    d = x[I] - x[J]
    r2 = (d * d).sum(1)
    dist = torch.sqrt(r2)
    s = torch.zeros(n, dtype=x.dtype, device=dev).index_add(0, I, _hct(dist, r2, r[I], r[J]))
    s = s.index_add(0, J, _hct(dist, r2, r[J], r[I]))
    born = 1 / torch.clamp(1 / r - 0.5 * s, min=2.0)
    # SASA: entries within reach, row by row in scan order
    R = r + 1.4
    with torch.no_grad():
        k = torch.nonzero(dist < R[I] + R[J]).reshape(-1)
        k = k[torch.argsort(I[k] * n + rank[J[k]])]
        start = torch.searchsorted(I[k].contiguous(), torch.arange(n, device=dev))
        col = torch.arange(len(k), device=dev) - start[I[k]]
        width = int(col.max()) + 1 if len(k) else 0
    cap = 2 * math.pi * R[I[k]] ** 2 * ((R[I[k]] + R[J[k]] - dist[k]) / (2 * R[I[k]]))
    padded = torch.zeros((width, n), dtype=x.dtype, device=dev).index_put((col, I[k]), cap)
    sa = 4 * math.pi * R * R
    for w in range(width):
        sa = sa - torch.minimum(0.85 * sa, padded[w])  # a padded entry takes 0
    sasa = 0.92 + 0.00542 * torch.clamp(sa, min=0).sum()
    # pairs
    with torch.no_grad():
        ptr = as_t(flat.excl_ptr, torch.long)
        ei = torch.repeat_interleave(torch.arange(n, device=dev), ptr[1:] - ptr[:-1])
        excl = torch.sort(ei * n + as_t(flat.excl_cols, torch.long)).values
        at = torch.searchsorted(excl, I * n + J).clamp(max=max(0, len(excl) - 1))
        bonded = excl[at] == I * n + J if len(excl) else torch.zeros_like(I, dtype=torch.bool)
        k = torch.nonzero(~bonded & (r2 <= 144.0)).reshape(-1)
    I, J, r2, dist = I[k], J[k], r2[k], dist[k]
    qq, sig, aa = q[I] * q[J], r[I] + r[J], born[I] * born[J]
    pair = 332.0636 / 78.5 * qq / dist * torch.exp(-0.1257 * dist)
    pair = pair - 0.5 * (1 - 1 / 78.5) * 332.0636 * qq / torch.sqrt(r2 + aa * torch.exp(-r2 / (4 * aa)))
    s6 = (sig * sig / r2) ** 3
    pair = pair + 4 * torch.sqrt(e[I] * e[J]) * (s6 * s6 - s6)
    t12 = (0.36 * sig * sig / r2) ** 6
    pair = pair + torch.where(dist < 0.6 * sig, torch.clamp(1e4 * (t12 - 1) ** 2, max=5e3), torch.zeros_like(r2))
    pair = pair.sum()
    # dihedral records and disulfides
    dih = torch.zeros((), dtype=x.dtype, device=dev)
    abcd = as_t(flat.dih_abcd, torch.long).reshape(-1, 4)
    if len(abcd):
        A, B, C, D = (x[abcd[:, c]] for c in range(4))
        b1, b2, b3 = A - B, C - B, D - C
        n1, n2 = torch.linalg.cross(b1, b2), torch.linalg.cross(b2, b3)
        phi = torch.atan2((torch.linalg.cross(n1, b2) * n2).sum(1), (n1 * n2).sum(1))
        off = as_t(flat.term_off, torch.long)
        rec = torch.repeat_interleave(torch.arange(len(abcd), device=dev), off[1:] - off[:-1])
        dih = (as_t(flat.term_v2) * (1 + torch.cos(as_t(flat.term_n) * phi[rec] - as_t(flat.term_gamma)))).sum()
    ss = torch.zeros((), dtype=x.dtype, device=dev)
    if len(flat.ss):
        p = as_t(flat.ss, torch.long).reshape(-1, 2)
        ss = (600.0 * ((x[p[:, 0]] - x[p[:, 1]]).norm(dim=1) - 2.044) ** 2).sum()
    return torch.stack([sasa, dih, ss, pair, sasa + dih + ss + pair])


def exact(case, seed):
    kind = case["kind"]
    if kind == "contacts":
        x = prepare(case, seed)["coords"]
        mean = torch.zeros((x.shape[1], x.shape[1]), dtype=torch.float64, device=x.device)
        near = torch.zeros_like(mean)
        for s in x:
            d2 = ((s[:, None, :] - s[None, :, :]) ** 2).sum(2)
            mean += torch.sqrt(d2)
            near += (d2 < 64.0).double()
        near.fill_diagonal_(0.0)
        return {"mean": mean / len(x), "contacts": near / len(x)}
    if kind not in ("score", "rescore", "forces"):
        return None  # a sampled chain: its accept decisions have no 64-bit value of their own
    rng = np.random.default_rng(seed)
    xyz, q, r, e, topo = _chain(case["residues"])
    x, flat = _coords(xyz, rng), flatten(topo)
    if kind == "score":
        return _exact_energy(torch.as_tensor(x, device="cuda"), q, r, e, flat).cpu().numpy()
    if kind == "rescore":
        with torch.no_grad():
            return torch.stack([_exact_energy(torch.as_tensor(f, device="cuda"), q, r, e, flat)
                                for f in _frames(x, case["frames"], rng)])
    p = torch.as_tensor(x, device="cuda").requires_grad_()
    terms = _exact_energy(p, q, r, e, flat)
    (grad,) = torch.autograd.grad(terms[4], p)
    if case["api"] == "autograd":
        return {"energy": terms[4:].detach(), "grad": grad}
    return {"terms": terms.detach().reshape(1, 5), "grad": torch.cat([grad, torch.zeros_like(grad[:, :1])], 1)}
