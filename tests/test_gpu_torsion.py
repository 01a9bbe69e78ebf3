"""GPU checks of torsion space: all-bond moves, the torsion gradient,
descent minimisation, MALA and the autograd wrapper (through the C ABI).

  * alma_torsion_apply vs the reference's one-bond-at-a-time rotations
    (numpy, axes from the updated coordinates): 1e-9 Å;
  * alma_torsion_grad vs the projection of the FP64 torch-autograd gradient
    (oracle/torch_energy.py) onto each bond: 1e-8 relative; and vs central
    finite differences of the energy (h = 1e-5 rad, list fixed) for bonds
    whose rotation moves no pair across the reference's 12 Å cutoff:
    1e-5 relative + 1e-6;
  * descent: monotone, ends below the start, final energy = a fresh
    evaluation of the final coordinates;
  * MALA: the device's log acceptance ratio equals a host recomputation
    from the oracle energy and the autograd torsion gradient at the
    proposal; runs are reproducible from the seed.
"""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _rot(p, o, u, d):
    v = p - o
    c, s = np.cos(d), np.sin(d)
    return o + v * c + np.cross(u, v) * s + np.outer(v @ u, u) * (1 - c)


def _sequential(x0, T, flat, delta):
    xs = x0.copy()
    for k in range(flat.nrb):
        if delta[k] == 0.0:
            continue
        side = np.array(sorted(T.side_set(k)))
        o = xs[flat.rb_i[k]]
        u = xs[flat.rb_j[k]] - o
        u /= np.linalg.norm(u)
        xs[side] = _rot(xs[side], o, u, delta[k])
    return xs


def _golden_batch(name, precision="fp64"):
    from conftest import Golden
    from protein_physics_b200.device import DeviceBatch
    from protein_physics_b200.topology import flatten
    g = Golden(name)
    T = g.topology()
    flat = flatten(T)
    b = DeviceBatch([(g["xyz"], g["q"], g["r"], g["eps"], flat)], precision=precision)
    return g, T, flat, b


def test_torsion_apply_matches_sequential():
    from protein_physics_b200 import synth
    from protein_physics_b200.device import DeviceBatch
    from protein_physics_b200.topology import BondTopology, flatten
    from protein_physics_b200.torsion import TorsionSpace
    chains, topos, flats = [], [], []
    for seed, nres in ((5, 10), (6, 14)):
        ch = synth.chain(nres, seed)
        T = BondTopology()
        T.build(ch.resnames, ch.atomnames, ch.res_idx)
        chains.append(ch)
        topos.append(T)
        flats.append(flatten(T))
    b = DeviceBatch([(c.xyz, c.charge, c.radius, c.epsilon, f) for c, f in zip(chains, flats)])
    ts = TorsionSpace(b)
    rng = np.random.default_rng(1)
    delta = rng.normal(0, 0.2, ts.nrb)
    ts.apply(torch.as_tensor(delta, device="cuda"))
    for s in range(2):
        d = delta[b.rb_off_h[s]:b.rb_off_h[s + 1]]
        ref = _sequential(chains[s].xyz, topos[s], flats[s], d)
        assert np.abs(b.coords(s) - ref).max() < 1e-9
    # masked: system 0 only
    before = [b.coords(s).copy() for s in range(2)]
    mask = torch.tensor([1, 0], dtype=torch.uint8, device="cuda")
    ts.apply(torch.as_tensor(delta, device="cuda"), sys_mask=mask)
    assert np.array_equal(b.coords(1), before[1])
    assert not np.array_equal(b.coords(0), before[0])


def _autograd_gtheta(x, gx, flat, T):
    out = np.zeros(flat.nrb)
    for k in range(flat.nrb):
        side = np.array(sorted(T.side_set(k)))
        o = x[flat.rb_i[k]]
        u = x[flat.rb_j[k]] - o
        u /= np.linalg.norm(u)
        out[k] = np.sum(np.cross(u, x[side] - o) * gx[side])
    return out


def test_torsion_grad_vs_autograd_and_fd(oracle):
    from torch_energy import TorchEnergy
    from protein_physics_b200.torsion import TorsionSpace
    g, T, flat, b = _golden_batch("insulin")
    b.build_nl()
    b.energy_terms()
    ts = TorsionSpace(b)
    gth = ts.gtheta(b.forces()).cpu().numpy()[:flat.nrb]
    ptr, cols = oracle.nl_build(g["xyz"])
    _, gx = TorchEnergy(g["q"], g["r"], g["eps"], ptr, cols, flat).energy_and_grad(g["xyz"])
    ref = _autograd_gtheta(np.asarray(g["xyz"]), gx, flat, T)
    assert np.abs(gth - ref).max() <= 1e-8 * max(1.0, np.abs(ref).max())
    # finite differences along single torsions, list fixed
    x0 = np.asarray(g["xyz"], np.float64)
    I = np.repeat(np.arange(g.n), np.diff(ptr))
    h = 1e-5
    rng = np.random.default_rng(3)
    checked = 0
    for k in rng.permutation(flat.nrb):
        side = np.array(sorted(T.side_set(k)))
        if side.size > 40:
            continue
        xs = [_sequential(x0, T, flat, np.where(np.arange(flat.nrb) == k, d, 0.0)) for d in (h, -h)]
        inside = [(((xx[I] - xx[cols]) ** 2).sum(1) <= 144.0) for xx in [x0] + xs]
        if not (np.array_equal(inside[0], inside[1]) and np.array_equal(inside[0], inside[2])):
            continue  # a pair crosses the reference's 12 Å cutoff: E jumps
        Es = []
        for xx in xs:
            b.xyz[:g.n, :3].copy_(torch.as_tensor(xx, device="cuda"))
            b.nl_ready = True  # same list: displacements are far inside the skin
            Es.append(float(b.energy_terms()[0, 4]))
        fd = (Es[0] - Es[1]) / (2 * h)
        assert abs(gth[k] - fd) <= 1e-5 * abs(fd) + 1e-6, (k, gth[k], fd)
        checked += 1
        if checked == 24:
            break
    assert checked >= 8


def test_minimize_monotone():
    from protein_physics_b200 import synth
    from protein_physics_b200.device import DeviceBatch
    from protein_physics_b200.topology import BondTopology, flatten
    from protein_physics_b200.torsion import minimize
    ch = synth.chain(24, 11)
    T = BondTopology()
    T.build(ch.resnames, ch.atomnames, ch.res_idx)
    b = DeviceBatch([(ch.xyz, ch.charge, ch.radius, ch.epsilon, flatten(T))], precision="mixed")
    hist, eta = minimize(b, steps=60)
    E = hist[:, 0].cpu().numpy()
    assert np.all(np.diff(E) <= 0.0)
    assert E[-1] < E[0]
    b.nl_ready = False
    assert float(b.energy_terms()[0, 4]) == pytest.approx(E[-1], rel=1e-12)


def test_mala_log_alpha_matches_host(oracle):
    from oracle import TopoArrays
    from torch_energy import TorchEnergy
    from protein_physics_b200.torsion import MALARunner
    g, T, flat, b = _golden_batch("insulin")
    x0 = np.asarray(g["xyz"], np.float64).copy()
    R = MALARunner(b, 0.6, seed=99, step=np.radians(0.5))
    st0 = R.state()
    g0 = R.cur.g.cpu().numpy()[:flat.nrb].copy()
    R.step()
    st1 = R.state()
    delta = R.delta.cpu().numpy()[:flat.nrb]
    sig = R.sigma.cpu().numpy()[:flat.nrb] * st0["scale"][0]  # the proposal's sigma (scale 1 at the start)
    x1 = _sequential(x0, T, flat, delta)
    E0 = oracle.calculate_potential(x0, g["q"], g["r"], g["eps"], TopoArrays(flat))[4]
    E1_host = oracle.calculate_potential(x1, g["q"], g["r"], g["eps"], TopoArrays(flat))[4]
    E1 = float(R.new.terms[0, 4].item())  # the device's energy at its own x1
    assert st0["energy"][0] == pytest.approx(E0, rel=1e-10)
    # The list grid starts one cell below the lowest coordinate, so the
    # extreme atom of each axis sits on a cell face and the last bit of its
    # coordinate picks the cell.  The host's sequential rotations and the
    # device's composed ones differ by ~1e-14 A, which can reorder that
    # atom's row and shift the order-dependent SASA sum by ~1e-5 kcal/mol
    # (the oracle itself shows it under 1e-13 A noise).  Same coordinates,
    # same energy: checked on the accepted state below.
    assert E1 == pytest.approx(E1_host, rel=1e-8)
    ptr, cols = oracle.nl_build(x1)
    _, gx1 = TorchEnergy(g["q"], g["r"], g["eps"], ptr, cols, flat).energy_and_grad(x1)
    g1 = _autograd_gtheta(x1, gx1, flat, T)
    beta = 1.0 / 0.6
    m = sig > 0
    sg = sig[m]

    c = R.cfg.drift_clip

    def drift(g):  # truncated at ±drift_clip·sigma
        return np.clip(-0.5 * sg ** 2 * beta * g, -c * sg, c * sg)
    fwd = np.sum((delta[m] - drift(g0[m])) ** 2 / (2 * sg ** 2))
    rev = np.sum((-delta[m] - drift(g1[m])) ** 2 / (2 * sg ** 2))
    la = -beta * (E1 - E0) - rev + fwd
    assert st1["log_alpha"][0] == pytest.approx(la, rel=1e-7, abs=1e-6)
    acc = bool(R.accept.cpu().numpy()[0])
    assert st1["n_accepted"][0] == int(acc)
    assert np.abs(b.coords(0) - (x1 if acc else x0)).max() < 1e-9
    if acc:
        E_dev_xyz = oracle.calculate_potential(b.coords(0), g["q"], g["r"], g["eps"], TopoArrays(flat))[4]
        assert st1["energy"][0] == pytest.approx(E_dev_xyz, rel=1e-10)


def test_mala_reproducible_and_mixing():
    from protein_physics_b200 import synth
    from protein_physics_b200.device import DeviceBatch
    from protein_physics_b200.topology import BondTopology, flatten
    from protein_physics_b200.torsion import MALARunner, minimize
    ch = synth.chain(16, 4)
    T = BondTopology()
    T.build(ch.resnames, ch.atomnames, ch.res_idx)
    flat = flatten(T)
    out = []
    for _ in range(2):
        b = DeviceBatch([(ch.xyz, ch.charge, ch.radius, ch.epsilon, flat)] * 2, precision="mixed")
        minimize(b, steps=100)
        R = MALARunner(b, [0.5962, 0.9], seed=5, step=np.radians(0.5))
        st = R.run(40)
        out.append((st, b.coords(0), b.coords(1)))
    assert np.array_equal(out[0][1], out[1][1]) and np.array_equal(out[0][2], out[1][2])
    st = out[0][0]
    assert np.all(st["n_proposed"] == 40)
    assert np.all(st["n_accepted"] > 0) and np.all(st["n_accepted"] < 40)


def test_autograd_energy_matches_forces():
    from protein_physics_b200.autograd import EnergyModel
    from protein_physics_b200.topology import flatten
    from conftest import Golden
    systems = []
    for n in ("insulin", "synth64"):
        g = Golden(n)
        systems.append((g["xyz"], g["q"], g["r"], g["eps"], flatten(g.topology())))
    model = EnergyModel(systems, precision="fp64")
    x = model.coords().requires_grad_()
    E = model(x)
    w = torch.tensor([2.0, -0.5], dtype=torch.float64, device="cuda")
    (E * w).sum().backward()
    b = model.batch
    f = b.forces()[:b.natoms, :3]
    sys_of = b.atom_sys
    assert torch.allclose(x.grad, f * w[sys_of].unsqueeze(1), rtol=0, atol=0)
    for s, (xyz, q, r, e, flat) in enumerate(systems):
        from protein_physics_b200.device import DeviceBatch
        ref = float(DeviceBatch([(xyz, q, r, e, flat)], precision="fp64").energy_terms()[0, 4])
        assert float(E[s].detach()) == pytest.approx(ref, rel=1e-13)


def test_mala_graph_replay_equals_eager():
    """One captured CUDA graph per proposal gives the eager chain bit for bit."""
    from protein_physics_b200 import synth
    from protein_physics_b200.device import DeviceBatch
    from protein_physics_b200.topology import BondTopology, flatten
    from protein_physics_b200.torsion import MALARunner, minimize
    ch = synth.chain(16, 4)
    T = BondTopology()
    T.build(ch.resnames, ch.atomnames, ch.res_idx)
    flat = flatten(T)
    out = []
    for graph in (False, True):
        b = DeviceBatch([(ch.xyz, ch.charge, ch.radius, ch.epsilon, flat)] * 2, precision="mixed")
        minimize(b, steps=50)
        R = MALARunner(b, [0.5962, 0.9], seed=8, step=np.radians(0.5))
        st = R.run(70, graph=graph, chunk=32)
        out.append((st, b.coords(0), b.coords(1)))
    assert np.array_equal(out[0][1], out[1][1]) and np.array_equal(out[0][2], out[1][2])
    for k in ("energy", "n_accepted", "n_proposed", "step", "scale"):
        assert np.array_equal(out[0][0][k], out[1][0][k]), k


@pytest.mark.parametrize("residues", [(16, 5, 31), (62, 63, 64, 65), (170,), (300,), (620,)])
def test_torsion_tiles_and_clusters(residues):
    """Chains whose atoms end inside, at and past a tile of the prefix sums,
    and whose bond counts take each cluster size: the torsion gradient of a
    random field and the all-bond move against numpy."""
    from conftest import ROOT
    from protein_physics_b200.device import DeviceBatch
    from protein_physics_b200.topology import BondTopology, flatten
    from protein_physics_b200.torsion import TorsionSpace
    w = np.load(os.path.join(ROOT, "workloads", "c4_globule_1000res.npz"), allow_pickle=False)
    ridx, systems, topos = w["res_idx"], [], []
    for k, n in enumerate(residues):
        r0 = 40 * k
        a, b_ = np.searchsorted(ridx, [r0, r0 + n])
        T = BondTopology()
        T.build([str(v) for v in w["resnames"][a:b_]], [str(v) for v in w["atomnames"][a:b_]],
                [int(v) - r0 for v in ridx[a:b_]])
        topos.append(T)
        systems.append((w["xyz"][a:b_].astype(np.float64), w["charge"][a:b_], w["radius"][a:b_], w["epsilon"][a:b_],
                        flatten(T)))
    b = DeviceBatch(systems)
    ts = TorsionSpace(b)
    rng = np.random.default_rng(7)
    grad = np.zeros((b.natoms, 4))
    grad[:, :3] = rng.normal(0, 10.0, (b.natoms, 3))
    gth = ts.gtheta(torch.as_tensor(grad, device="cuda")).cpu().numpy()
    delta = rng.normal(0, 0.05, ts.nrb)
    ts.apply(torch.as_tensor(delta, device="cuda"))
    for s, (x, _, _, _, flat) in enumerate(systems):
        k0, k1, a0 = b.rb_off_h[s], b.rb_off_h[s + 1], b.atom_off_h[s]
        ref = _autograd_gtheta(x, grad[a0:a0 + flat.n, :3], flat, topos[s])
        # sums of up to n torques of size |x| |g|, in FP64
        assert np.abs(gth[k0:k1] - ref).max() <= 1e-13 * flat.n * 100.0 * 10.0
        assert np.abs(b.coords(s) - _sequential(x, topos[s], flat, delta[k0:k1])).max() < 1e-9


def _run_of_residues(name, residues, r0=0):
    """(system, topology) of a run of residues of a benchmark chain."""
    from conftest import ROOT
    from protein_physics_b200.topology import BondTopology, flatten
    w = np.load(os.path.join(ROOT, "workloads", name + ".npz"), allow_pickle=False)
    ridx = w["res_idx"]
    a, b = np.searchsorted(ridx, [r0, r0 + residues])
    T = BondTopology()
    T.build([str(v) for v in w["resnames"][a:b]], [str(v) for v in w["atomnames"][a:b]],
            [int(v) - r0 for v in ridx[a:b]])
    return (w["xyz"][a:b].astype(np.float64), w["charge"][a:b], w["radius"][a:b], w["epsilon"][a:b], flatten(T)), T


def test_torsion_apply_of_uneven_batches():
    """A chain of far more bonds than the mean (1,000 and more past what a CTA
    of the batch's launch holds) is turned by a launch of its own: to the bit as
    alone, first or last in the batch, masked or not."""
    from protein_physics_b200.device import DeviceBatch
    from protein_physics_b200.torsion import TorsionSpace
    long, _ = _run_of_residues("c4_globule_1000res", 500)
    short = [_run_of_residues("c4_globule_1000res", 6 + k % 5, 7 * k)[0] for k in range(40)]
    rng = np.random.default_rng(2)
    delta = [rng.normal(0, 0.05, s[4].nrb) for s in [long] + short]
    alone = []
    for s, d in zip([long] + short, delta):
        b = DeviceBatch([s])
        TorsionSpace(b).apply(torch.as_tensor(d, device="cuda"))
        alone.append(b.coords(0))
    for order in (list(range(41)), list(range(40, -1, -1))):
        systems = [([long] + short)[k] for k in order]
        assert sum(s[4].nrb for s in systems) / 41 < 512 < 1024 < long[4].nrb
        for mask in (None, torch.tensor([k % 2 for k in order], dtype=torch.uint8, device="cuda")):
            b = DeviceBatch(systems)
            before = [b.coords(p) for p in range(41)]
            TorsionSpace(b).apply(torch.as_tensor(np.concatenate([delta[k] for k in order]), device="cuda"),
                                  sys_mask=mask)
            for p, k in enumerate(order):
                assert np.array_equal(b.coords(p), alone[k] if mask is None or k % 2 else before[p]), (p, k)


def test_torsion_apply_past_the_shared_memory():
    """A chain of more bonds than a cluster's shared memory holds (8 x 1,024)
    takes the global buffers: 40 of its bonds turned, against numpy."""
    from protein_physics_b200.device import DeviceBatch
    from protein_physics_b200.torsion import TorsionSpace
    system, T = _run_of_residues("c5_multidomain_4x1000res", 4030)
    flat = system[4]
    assert flat.nrb > 8 * 1024
    rng = np.random.default_rng(6)
    delta = np.zeros(flat.nrb)
    delta[rng.choice(flat.nrb, 40, replace=False)] = rng.normal(0, 0.05, 40)
    b = DeviceBatch([system])
    TorsionSpace(b).apply(torch.as_tensor(delta, device="cuda"))
    assert np.abs(b.coords(0) - _sequential(system[0], T, flat, delta)).max() < 1e-9


def test_torsion_grad_of_any_side_list():
    """Sides given as atom lists of every length class (none, one share of eight
    lanes, several, more than a warp), with and without a range, in two systems
    whose bond counts fill no block: against numpy.  Sums of up to n torques
    |x| |g|, in FP64."""
    import ctypes as C
    import dataclasses
    from protein_physics_b200 import _lib
    from protein_physics_b200.device import DeviceBatch, _empty_topo, _ptr
    rng = np.random.default_rng(12)
    systems, sides = [], []
    for n, nrb in ((130, 37), (90, 5)):
        explicit = [np.sort(rng.choice(n, min(n, k), replace=False)).astype(np.int32)
                    for k in ([0, 1, 7, 8, 9, 16, 17, 24, 31, 32, 33, 64, 70] * 3)[:nrb]]
        lo = np.where(np.arange(nrb) % 3 == 0, 0, rng.integers(0, n // 2, nrb))
        hi = np.where(np.arange(nrb) % 3 == 0, 0, rng.integers(n // 2, n + 1, nrb))
        ij = np.stack([rng.choice(n, 2, replace=False) for _ in range(nrb)])
        flat = dataclasses.replace(
            _empty_topo(n), rb_i=ij[:, 0].astype(np.int32), rb_j=ij[:, 1].astype(np.int32),
            rb_kind=np.zeros(nrb, np.int32), rb_scale=np.ones(nrb),
            side_ptr=np.concatenate([[0], np.cumsum([len(e) for e in explicit])]).astype(np.int64),
            side_idx=np.concatenate(explicit), side_lo=lo.astype(np.int32), side_hi=hi.astype(np.int32),
            side_count=np.array([len(e) + h - l for e, l, h in zip(explicit, lo, hi)], np.int64))
        systems.append((rng.uniform(0, 30, (n, 3)), np.zeros(n), np.full(n, 1.5), np.zeros(n), flat))
        sides.append([np.concatenate([e, np.arange(l, h)]).astype(int) for e, l, h in zip(explicit, lo, hi)])
    b = DeviceBatch(systems)
    grad = np.zeros((b.natoms, 4))
    grad[:, :3] = rng.normal(0, 10.0, (b.natoms, 3))
    nrb = int(b.rb_off_h[-1])
    ws = torch.zeros(b.L.alma_torsion_workspace_bytes(b.natoms, b.nsys, nrb), dtype=torch.uint8, device="cuda")
    g, out = torch.as_tensor(grad, device="cuda"), torch.zeros(nrb, dtype=torch.float64, device="cuda")
    _lib.check(b.L.alma_torsion_grad(C.byref(b.batch_s), C.byref(b.topo_s), _ptr(g), None, _ptr(ws), _ptr(out),
                                     b._sp()), "alma_torsion_grad")
    out = out.cpu().numpy()
    for s, (x, _, _, _, flat) in enumerate(systems):
        gs = grad[b.atom_off_h[s]:b.atom_off_h[s + 1], :3]
        for k in range(flat.nrb):
            u = x[flat.rb_j[k]] - x[flat.rb_i[k]]
            ref = np.sum(np.cross(u / np.linalg.norm(u), x[sides[s][k]] - x[flat.rb_i[k]]) * gs[sides[s][k]])
            assert abs(out[b.rb_off_h[s] + k] - ref) <= 1e-13 * 2 * flat.n * 52.0 * 40.0, (s, k)
