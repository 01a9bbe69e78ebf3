"""GPU parity: the sm_100a kernels (through the C ABI) against the oracle
and the reference's golden vectors.

Bars (the reference's own path is FP64):
  * neighbor lists, exclusion flags: bit-exact, row order included;
  * FP64 mode: energies 1e-10 relative, Born radii 1e-12 relative,
    move ΔE 1e-7 kcal/mol absolute (summation order differs only);
  * mixed mode (FP32 pair terms, FP64 accumulation): total energy 1e-6
    relative; move ΔE 1e-4 kcal/mol absolute on the PDB systems.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _batch(golden, precision="mixed", topo=True):
    from protein_physics_b200.device import DeviceBatch
    from protein_physics_b200.topology import flatten
    flat = flatten(golden.topology()) if topo else None
    return DeviceBatch([(golden["xyz"], golden["q"], golden["r"], golden["eps"], flat)], precision=precision)


def test_nl_bit_exact(golden, oracle):
    b = _batch(golden)
    b.build_nl()
    rp, cols, flags = b.nl_host(0, half=True)
    ptr, ocols = oracle.nl_build(golden["xyz"])
    assert np.array_equal(rp, ptr)
    assert np.array_equal(cols, ocols)  # row order included (SASA depends on it)
    # exclusion flags = the topology's exclusion test
    from oracle import TopoArrays
    from protein_physics_b200.topology import flatten
    T = golden.topology()
    ex = np.array([T.is_excluded(i, int(j)) for i in range(golden.n) for j in ocols[ptr[i]:ptr[i + 1]]], np.uint8)
    assert np.array_equal(flags, ex)
    # full rows: both directions, same sets
    frp, fcols, _ = b.nl_host(0, half=False)
    for i in range(0, golden.n, max(1, golden.n // 97)):
        half_i = set(ocols[ptr[i]:ptr[i + 1]].tolist())
        lower = {k for k in range(i) if i in set(ocols[ptr[k]:ptr[k + 1]].tolist())}
        assert set(fcols[frp[i]:frp[i + 1]].tolist()) == half_i | lower


def test_nl_short_rows(golden):
    """Short rows: the full/half rows filtered, in order, to the pairs within
    R*_i + R*_j + 2 probe + skin (+1e-6) at build time."""
    b = _batch(golden)
    b.build_nl()
    p = b.params
    pad = 2.0 * p.probe_r + 2.0 * np.sqrt(p.half_skin2) + 1e-6
    x, r = golden["xyz"], golden["r"]
    for half in (True, False):
        rp, cols, flags = b.nl_host(0, half=half)
        srp, scols, sflags = b.nl_host(0, half=half, short=True)
        for i in range(golden.n):
            row = cols[rp[i]:rp[i + 1]]
            fl = flags[rp[i]:rp[i + 1]]
            reach = r[i] + pad + r[row]
            keep = np.sum((x[row] - x[i]) ** 2, axis=1) < reach * reach
            assert np.array_equal(scols[srp[i]:srp[i + 1]], row[keep]), i
            assert np.array_equal(sflags[srp[i]:srp[i + 1]], fl[keep]), i
    need = b.need.cpu().numpy()[0]
    assert need[2] == len(b.nl_host(0, half=False, short=True)[1])
    assert need[3] == len(b.nl_host(0, half=True, short=True)[1])


@pytest.mark.parametrize("precision,rtol", [("fp64", 1e-12), ("mixed", 2e-6)])
def test_born_radii(golden, oracle, precision, rtol):
    b = _batch(golden, precision)
    b.build_nl()
    b.born_radii()
    a = b.born[:golden.n].cpu().numpy()
    np.testing.assert_allclose(a, golden["born"], rtol=rtol, atol=0)


@pytest.mark.parametrize("precision,rtol", [("fp64", 1e-10), ("mixed", 1e-6)])
def test_energy_terms(golden, precision, rtol):
    b = _batch(golden, precision)
    terms = b.energy_terms()[0].cpu().numpy()
    ref = golden["energy_topo"]
    assert abs(terms[4] - ref[4]) <= rtol * abs(ref[4])
    np.testing.assert_allclose(terms[:3], ref[:3], rtol=1e-10, atol=1e-9)  # SASA/dihedral/SS are FP64 always
    b2 = _batch(golden, precision, topo=False)
    t2 = b2.energy_terms()[0].cpu().numpy()
    assert abs(t2[4] - golden["energy_notopo"][4]) <= rtol * abs(golden["energy_notopo"][4])


def test_bridge_case():
    import json
    import os
    from conftest import GOLDEN
    from protein_physics_b200 import Particle, PhysicsEngine
    g = json.load(open(os.path.join(GOLDEN, "bridge.json")))
    P = [Particle(*x, q) for x, q in zip(g["xyz"], g["q"])]
    assert PhysicsEngine(precision="fp64").calculate_potential(P) == pytest.approx(g["energy"], rel=1e-12)
    assert PhysicsEngine().calculate_potential(P) == pytest.approx(g["energy"], rel=1e-6)


def _move_args(golden, T, kind, code):
    if kind == 0:
        return 0, int(code)
    phi_k, psi_k = divmod(int(code), 100000)
    return 1, sorted(T.concerted_pairs).index((phi_k, psi_k))


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_move_dE_vs_reference(golden, precision):
    T = golden.topology()
    b = _batch(golden, precision)
    b.build_nl()
    b.born_radii()
    errs = []
    for kind, code, delta, dE_ref, *terms_ref in golden["moves"]:
        k, a = _move_args(golden, T, int(kind), code)
        dE, dterms = b.move_dE([k], [a], [[delta, 0.0]])
        dE = float(dE[0].item())
        dterms = dterms[0].cpu().numpy()
        if precision == "fp64":
            assert dE == pytest.approx(dE_ref, abs=1e-7 + 1e-12 * abs(dE_ref))
            np.testing.assert_allclose(dterms, terms_ref, atol=1e-7, rtol=1e-12)
        else:
            # 1e-4 kcal/mol; plus the FP64 rounding floor of the reference's
            # own sums when a move carries a clash of ~1e11 kcal/mol
            scale = np.sum(np.abs(terms_ref))
            tol = 1e-4 + 1e-14 * scale
            assert abs(dE - dE_ref) <= tol, (kind, code, dE, dE_ref)
            np.testing.assert_allclose(dterms[1:], terms_ref[1:], atol=1e-8, rtol=1e-11)  # SASA/dih/SS FP64
        errs.append(abs(dE - dE_ref))
    # the state must be unchanged after non-applied proposals
    assert np.array_equal(b.coords(0), golden["xyz"])


def test_move_apply_matches_oracle(golden, oracle):
    from oracle import TopoArrays
    from protein_physics_b200.topology import flatten
    T = golden.topology()
    flat = flatten(T)
    b = _batch(golden, "fp64")
    b.build_nl()
    b.born_radii()
    x, q, r, e = golden["xyz"], golden["q"], golden["r"], golden["eps"]
    nl = oracle.nl_build(x)
    a = oracle.born_radii(x, r, nl)
    k = int(np.argmax([len(s) for s in T.rot_bond_sides]) // 2)
    side = T.rot_bond_sides[k]
    group = np.zeros(golden.n, np.int8)
    group[side] = 1
    dE_o, _, new_xyz, new_a = oracle.move_dE(x, q, r, e, nl, a, TopoArrays(flat), [(T.rot_bonds[k].i, T.rot_bonds[k].j,
                                                                                    0.2, side)], group)
    dE, _ = b.move_dE([0], [k], [[0.2, 0.0]], apply=True)
    assert float(dE[0]) == pytest.approx(dE_o, abs=1e-7)
    np.testing.assert_allclose(b.coords(0), new_xyz, rtol=0, atol=1e-12)
    np.testing.assert_allclose(b.born[:golden.n].cpu().numpy(), new_a, rtol=1e-12, atol=0)


def test_batched_equals_single():
    from conftest import Golden
    from protein_physics_b200.device import DeviceBatch
    from protein_physics_b200.topology import flatten
    gs = [Golden(n) for n in ("xq8", "insulin", "synth64")]
    systems = [(g["xyz"], g["q"], g["r"], g["eps"], flatten(g.topology())) for g in gs]
    B = DeviceBatch(systems)
    tb = B.energy_terms().cpu().numpy()
    for s, sysd in enumerate(systems):
        S = DeviceBatch([sysd])
        ts = S.energy_terms().cpu().numpy()[0]
        assert np.array_equal(ts, tb[s])  # bit-identical: same per-atom work, same reduction order
        rp_b, c_b, f_b = B.nl_host(s)
        rp_s, c_s, f_s = S.nl_host(0)
        assert np.array_equal(rp_b, rp_s) and np.array_equal(c_b, c_s) and np.array_equal(f_b, f_s)


def test_deterministic():
    from conftest import Golden
    g = Golden("xq8")
    r1 = _batch(g).energy_terms().cpu().numpy()
    r2 = _batch(g).energy_terms().cpu().numpy()
    assert np.array_equal(r1, r2)


def test_dropin_api(golden):
    from protein_physics_b200 import Particle, PhysicsEngine
    P = [Particle(*x, q, r, e) for x, q, r, e in zip(golden["xyz"], golden["q"], golden["r"], golden["eps"])]
    eng = PhysicsEngine()
    E = eng.calculate_potential(P, golden.topology())
    assert E == pytest.approx(golden["energy_topo"][4], rel=1e-6)
    assert eng.calculate_potential(P) == pytest.approx(golden["energy_notopo"][4], rel=1e-6)
    assert eng.calculate_potential([]) == 0.0
    assert "B200" in PhysicsEngine.device_name() or len(PhysicsEngine.device_name()) > 0


def test_engine_reuses_batch_across_calls(golden):
    """Repeated calls on one system reuse the device batch (coordinates
    reloaded): energies equal a fresh engine's, also after the coordinates
    change, and a different parameter set gets its own batch."""
    from protein_physics_b200 import Particle, PhysicsEngine
    T = golden.topology()
    eng = PhysicsEngine()
    P = [Particle(*x, q, r, e) for x, q, r, e in zip(golden["xyz"], golden["q"], golden["r"], golden["eps"])]
    E1 = eng.calculate_potential(P, T)
    x2 = np.asarray(golden["xyz"]) + np.random.default_rng(2).normal(0, 0.05, (golden.n, 3))
    P2 = [Particle(*x, q, r, e) for x, q, r, e in zip(x2, golden["q"], golden["r"], golden["eps"])]
    E2 = eng.calculate_potential(P2, T)
    assert len(eng._batches) == 1
    assert E2 == PhysicsEngine().calculate_potential(P2, T)
    assert eng.calculate_potential(P, T) == E1
    P3 = [Particle(*x, 0.5 * q, r, e) for x, q, r, e in zip(golden["xyz"], golden["q"], golden["r"], golden["eps"])]
    assert eng.calculate_potential(P3, T) == PhysicsEngine().calculate_potential(P3, T)
    assert len(eng._batches) == 2


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_row_spans_and_edge_skip(golden, precision):
    """AlmaNL.full_span holds each full row's smallest and largest atom
    index, and a move gives the same ΔE terms whether or not the kernels may
    skip the rows that move whole (no cross pair, no SASA mark in them):
    every torsion, crankshaft and concerted-pair move of the system."""
    T = golden.topology()
    on = _batch(golden, precision)
    off = _batch(golden, precision)
    off.set_row_spans(False)
    for b in (on, off):
        b.build_nl()
        b.born_radii()
    rp, cols, _ = on.nl_host(0, half=False)
    span = on.full_span[:golden.n].cpu().numpy()
    for i in range(golden.n):
        row = cols[rp[i]:rp[i + 1]]
        assert tuple(span[i]) == ((int(row.min()), int(row.max())) if row.size else (2 ** 31 - 1, -1))
    moves = [(0, k) for k in range(len(T.rot_bonds))]
    moves += [(1, k) for k in range(len(T.concerted_pairs))]
    moves += [(2, k) for k in range(len(T.concerted_sidechain_pairs))]
    rng = np.random.default_rng(5)
    tol = 1e-11 if precision == "fp64" else 1e-9
    inner = 0
    for kind, a in moves:
        d = rng.uniform(-0.3, 0.3, 2)
        e1, t1 = on.move_dE([kind], [a], [d])
        e0, t0 = off.move_dE([kind], [a], [d])
        t1, t0 = t1[0].cpu().numpy(), t0[0].cpu().numpy()
        np.testing.assert_allclose(t1, t0, rtol=tol, atol=1e-9, err_msg=str((kind, a)))
        assert float(e1[0]) == pytest.approx(float(e0[0]), rel=tol, abs=1e-9)
    # the skip engages: some torsion side holds atoms whose rows stay inside it
    from protein_physics_b200.topology import flatten
    F = flatten(T)
    for k in range(F.nrb):
        lo, hi = int(F.side_lo[k]), int(F.side_hi[k])
        inner += int(np.sum((span[lo:hi, 0] >= lo) & (span[lo:hi, 1] < hi)))
    assert inner > 0
    # commits of the largest sides (their inner members' Born radii come from
    # the commit pass): same coordinates, same radii
    big = np.argsort(-F.side_count)[:4]
    for kind, a in [(0, int(k)) for k in big] + [(1, 0)] * (len(T.concerted_pairs) > 0):
        for b in (on, off):
            b.move_dE([kind], [a], [[0.2, 0.0]], apply=True)
        assert np.array_equal(on.coords(0), off.coords(0))
        np.testing.assert_allclose(on.born[:golden.n].cpu().numpy(), off.born[:golden.n].cpu().numpy(),
                                   rtol=1e-12 if precision == "fp64" else 1e-6)


def test_nl_overflow_regrows_and_rebuilds(oracle):
    """Regions far too small for the rows: the build raises the overflow,
    the batch regrows its regions from need[] and builds again; the rows are
    then bit-exact, and a masked rebuild of one system after its atoms move
    leaves the other system's rows as they were."""
    from conftest import Golden
    from protein_physics_b200.device import DeviceBatch
    from protein_physics_b200.topology import flatten

    class Tight(DeviceBatch):
        NL_FULL_PER_ATOM = 1
        NL_HALF_PER_ATOM = 1
        NL_SHORT_PER_ATOM = 2

    gs = [Golden("insulin"), Golden("xq8")]
    systems = [(g["xyz"], g["q"], g["r"], g["eps"], flatten(g.topology())) for g in gs]
    b = Tight(systems)
    assert int(b.full_base[-1]) < 2 * b.natoms + 1000  # the initial regions cannot hold the rows
    b.build_nl()
    for s, g in enumerate(gs):
        rp, cols, _ = b.nl_host(s, half=True)
        ptr, ocols = oracle.nl_build(g["xyz"])
        assert np.array_equal(rp, ptr) and np.array_equal(cols, ocols), s
    before = b.nl_host(1, half=False)
    x = b.xyz.clone()
    a0, a1 = int(b.atom_off_h[0]), int(b.atom_off_h[1])
    x[a0:a1, :3] += 0.3
    b.xyz.copy_(x)
    mask = torch.tensor([1, 0], dtype=torch.uint8, device="cuda")
    b.build_nl(sys_mask=mask)
    after = b.nl_host(1, half=False)
    assert all(np.array_equal(u, v) for u, v in zip(before, after))
    rp, cols, _ = b.nl_host(0, half=True)
    ptr, ocols = oracle.nl_build(b.coords(0))
    assert np.array_equal(rp, ptr) and np.array_equal(cols, ocols)


def test_exclusion_window(golden):
    """alma_excl_window against its restatement from the CSR rows, and the
    list rows with the windows equal to those of the per-pair CSR search,
    flags and order included (insulin's disulfides take the far path)."""
    from conftest import excl_window_np
    from protein_physics_b200.device import _ptr
    b = _batch(golden)
    ref = excl_window_np(b.t_excl_ptr.cpu().numpy(), b.t_excl_cols.cpu().numpy(), b.natoms)
    got = b.t_excl_win.cpu().numpy().view(np.uint32).reshape(-1, 4)[:b.natoms]
    assert np.array_equal(got, ref)
    if len(golden.d["ss_in"]):
        assert (ref[:, 2] & 1).any()
    kinds = [(h, s) for h in (True, False) for s in (False, True)]
    b.build_nl()
    with_win = [b.nl_host(0, half=h, short=s) for h, s in kinds]
    b.topo_s.excl_win = None
    try:
        b.nl_ready = False
        b.build_nl()
        csr = [b.nl_host(0, half=h, short=s) for h, s in kinds]
    finally:
        b.topo_s.excl_win = _ptr(b.t_excl_win)
    for a, c in zip(with_win, csr):
        for x, y in zip(a, c):
            assert np.array_equal(x, y)


def _clouds(kind):
    rng = np.random.default_rng(11)
    if kind == "tiny":  # around a chunk, and a chain of one atom
        return [rng.uniform(0, 20, (n, 3)) for n in (1, 2, 31, 32, 33, 95)]
    if kind == "long rows":  # more neighbours than a row's stage, more chunks than its mask list
        return [rng.uniform(0, 11, (1400, 3)), rng.uniform(0, 60, (700, 3)), rng.uniform(0, 24, (5600, 3))]
    if kind == "stretched":  # a long thin box far from the origin: wide FP32 margins, mostly empty cells
        x = rng.uniform(0, 1, (3000, 3)) * [2500.0, 30.0, 20.0] + [4.0e4, -3.0e4, 10.0]
        return [x, rng.uniform(0, 25, (40, 3))]
    # two atoms per warp, uneven systems whose slots meet inside a warp
    return [rng.uniform(0, 18 + 4 * k, (1501 + 1200 * k, 3)) for k in range(6)]


@pytest.mark.parametrize("kind", ["tiny", "long rows", "stretched", "two per warp"])
def test_nl_rows_at_the_edges(oracle, kind):
    """Half rows equal to the oracle's, order included, and full rows the same
    pairs from both ends, where the build changes path."""
    from protein_physics_b200.device import DeviceBatch
    clouds = _clouds(kind)
    b = DeviceBatch([(x, np.zeros(len(x)), np.full(len(x), 1.9), np.full(len(x), 0.1), None) for x in clouds])
    assert kind != "two per warp" or b.natoms >= 24000
    b.build_nl()
    need = b.need.cpu().numpy()
    for s, x in enumerate(clouds):
        rp, cols, _ = b.nl_host(s, half=True)
        ptr, ocols = oracle.nl_build(x)
        assert np.array_equal(rp, ptr) and np.array_equal(cols, ocols), s
        frp, fcols, _ = b.nl_host(s, half=False)
        n = len(x)
        I = np.repeat(np.arange(n), np.diff(ptr))
        J = np.repeat(np.arange(n), np.diff(frp))
        both = np.concatenate([I * n + ocols, ocols.astype(np.int64) * n + I])
        assert np.array_equal(np.sort(J * n + fcols), np.sort(both)), s
        keep = fcols > J  # the full row holds the half row in its order
        assert np.array_equal(fcols[keep], ocols), s
        assert need[s, 0] == len(fcols) and need[s, 1] == len(ocols)


def _one_bond_system(xyz, q, r, eps, side):
    """A system of loose atoms and one rotatable bond 1-2 whose j-side is the
    atom range `side`."""
    import dataclasses
    from protein_physics_b200.device import _empty_topo
    flat = dataclasses.replace(
        _empty_topo(len(q)), rb_i=np.array([1], np.int32), rb_j=np.array([2], np.int32),
        rb_kind=np.array([2], np.int32), rb_scale=np.ones(1), side_ptr=np.zeros(2, np.int64),
        side_lo=np.array([side[0]], np.int32), side_hi=np.array([side[1]], np.int32),
        side_count=np.array([side[1] - side[0]], np.int64))
    return np.asarray(xyz, np.float64), np.asarray(q, np.float64), np.asarray(r, np.float64), \
        np.asarray(eps, np.float64), flat


def test_move_gb_change_of_far_pairs(oracle):
    """A pair whose distance stays while a Born radius changes: its GB energy
    changes by C qq (fo² - fn²) / (fo fn (fo + fn)), and fo² - fn² lies all in
    the exponentials A exp(-r²/4A), however far below the last bit of f² these
    are.  Atom 2 turns about its own axis: it stays where it is and takes its
    half-list radius, without the descreening by atoms 0 and 1; r² is 61-70
    times the larger A = a_0 a_2.  Tolerance: the argument r²/4A <= 17.5 is good
    to 4 x 2^-23 and the exponential to 22 x 2^-23 on top, 1.1e-5 of each term;
    the terms differ by a factor of 10 or more, the other factors are good to
    1e-6."""
    from protein_physics_b200.device import DeviceBatch
    r = np.array([0.42, 1.2, 0.35])
    systems = []
    for m in (61.0, 63.5, 66.0, 70.0):
        x = np.array([[3.0, 0.0, 0.0], [0.0, 0.0, 1.3], [0.0, 0.0, 0.0]])
        for _ in range(50):  # the radii depend a little on the distance
            a = oracle.born_radii(x, r, oracle.nl_build(x))
            x[0, 0] = np.sqrt(m * a[0] * a[2])
        systems.append(_one_bond_system(x, [1.0, 0.0, 1.0], r, np.zeros(3), (2, 3)))
    b = DeviceBatch(systems)
    b.build_nl()
    b.born_radii()
    a = b.born.cpu().numpy().reshape(-1, 3)
    d2 = np.array([s[0][0, 0] ** 2 for s in systems])
    Ao, An = a[:, 0] * a[:, 2], a[:, 0] * r[2]  # no atom follows atom 2: its half row is empty
    xo, xn = Ao * np.exp(-d2 / (4 * Ao)), An * np.exp(-d2 / (4 * An))
    assert np.all(a[:, 2] < 0.5) and np.all(xo > 10 * xn)
    assert np.all(d2 > 60.5 * Ao) and np.all(d2 < 70.5 * Ao)
    fo, fn = np.sqrt(d2 + xo), np.sqrt(d2 + xn)
    p = b.params
    gb = -0.5 * (1.0 / p.eps_prot - 1.0 / p.eps_water) * p.coulomb
    k = np.zeros(len(systems), int)
    _, terms = b.move_dE(k, k, np.full((len(systems), 2), 0.4))
    np.testing.assert_allclose(terms[:, 0].cpu().numpy(), gb * (xo - xn) / (fo * fn * (fo + fn)), rtol=1.5e-5)


def test_move_lj_outside_sigma_is_rounded_once():
    """LJ of a pair just outside sigma, where s² = sigma²/r² is an FP64
    quotient rounded to FP32: the quotients lie 1-4 FP64 ulps above the middle
    of two FP32 values, so that an approximate one falls to the other side.
    There 4 (s¹² - s⁶) changes by 12 for s², and an ulp of it (2^-24) is worth
    7e-7.  The moved atom goes to 11.5 Å, where the term is below 0.02 kcal/mol
    and its FP32 roundings are below 5 x 2^-24 of it, 6e-9."""
    from fractions import Fraction
    from protein_physics_b200.device import DeviceBatch
    rng = np.random.default_rng(3)
    f32 = np.float32
    systems, old = [], []
    while len(systems) < 64:
        r = float(rng.integers(3 << 20, 9 << 19)) / (1 << 20)  # r² exact
        lo = f32(rng.uniform(0.99993, 0.99998))
        mid = (float(lo) + float(np.nextafter(lo, f32(1)))) / 2
        sig = np.sqrt(mid * r * r)
        for _ in range(16):
            if sig * sig / (r * r) > mid:
                break
            sig = np.nextafter(sig, 10.0)
        s2 = sig * sig / (r * r)
        if not mid < s2 <= mid * (1 + 2.0 ** -50):
            continue
        u = f32(s2)
        s6 = f32(f32(u * u) * u)
        old.append(4.0 * float(f32(float(Fraction(float(s6)) ** 2 - Fraction(float(s6))))))
        cx = (r + 11.5) / 2  # half a turn about the axis through (cx, 0): r -> 11.5
        x = [[0.0, 0.0, 0.0], [cx, 0.0, -5.0], [cx, 0.0, -6.5], [r, 0.0, 0.0]]
        systems.append(_one_bond_system(x, np.zeros(4), [1.0, 0.01, 0.01, sig - 1.0], [1.0, 0.0, 0.0, 1.0], (3, 4)))
    b = DeviceBatch(systems)
    b.build_nl()
    b.born_radii()
    k = np.zeros(len(systems), int)
    _, terms = b.move_dE(k, k, np.full((len(systems), 2), np.pi))
    s6 = np.array([(s[2].sum() - 0.02) / 11.5 for s in systems]) ** 6
    np.testing.assert_allclose(terms[:, 0].cpu().numpy(), 4 * (s6 * s6 - s6) - np.array(old), rtol=0, atol=2e-8)


def _spread_system(extent, seed, n=24):
    """Atoms in two clumps at opposite corners of a box of `extent` Å."""
    rng = np.random.default_rng(seed)
    x = rng.uniform(0, 12, (n, 3))
    x[n // 2:] += extent
    return x, rng.choice([-0.4, 0.4], n), np.full(n, 1.7), np.full(n, 0.1), None


@pytest.mark.parametrize("rows", ["roomy", "tight"])
def test_nl_of_atoms_far_apart(oracle, rows):
    """Systems whose grids hold many times the cells that were allotted, alone
    or together with rows that do not fit: cells and rows are regrown in turn
    until the list is complete."""
    from protein_physics_b200.device import DeviceBatch

    class Tight(DeviceBatch):
        NL_FULL_PER_ATOM = 1
        NL_HALF_PER_ATOM = 1
        NL_SHORT_PER_ATOM = 2

    # rows far past the tight regions (one entry per atom and 64 more)
    rng = np.random.default_rng(4)
    dense = (rng.uniform(0, 30, (1400, 3)), np.zeros(1400), np.full(1400, 1.7), np.full(1400, 0.1), None)
    systems = [_spread_system(1000.0, 1), dense, _spread_system(40.0, 2), _spread_system(700.0, 3)]
    b = (Tight if rows == "tight" else DeviceBatch)(systems, precision="fp64")
    cells = [np.prod(np.ceil((np.ptp(s[0], axis=0) + 3 * 14.000001) / 14.000001)) for s in systems]
    assert sum(cells) > 16 * b.max_cells
    terms = b.energy_terms().cpu().numpy()
    for s, (x, q, r, e, _) in enumerate(systems):
        rp, cols, _ = b.nl_host(s, half=True)
        ptr, ocols = oracle.nl_build(x)
        assert np.array_equal(rp, ptr) and np.array_equal(cols, ocols), s
        assert terms[s, 4] == pytest.approx(oracle.calculate_potential(x, q, r, e)[4], rel=1e-10)


def test_nl_that_cannot_be_built_raises():
    """A box with more cells than the list can index is an error, not a list
    without pairs; the batch works again with coordinates that fit."""
    from protein_physics_b200.device import DeviceBatch
    x, q, r, e, _ = _spread_system(1.0e6, 5)
    b = DeviceBatch([(x, q, r, e, None)])
    with pytest.raises(RuntimeError, match="neighbor list"):
        b.energy_terms()
    with pytest.raises(RuntimeError, match="neighbor list"):
        b.evaluate()
    near = _spread_system(5.0, 5)
    b.load_coords(near[0])
    want = DeviceBatch([near]).energy_terms()
    assert torch.equal(b.energy_terms(), want)


def test_terms_of_many_small_systems_equal_each_alone():
    """Many small systems are summed by a CTA each, one alone by a cluster of
    eight: the same shares in the same order, so the same bits, with atom
    counts on both sides of a share (256) and of a round of shares (2,048)."""
    from conftest import Golden
    from protein_physics_b200.device import DeviceBatch
    from protein_physics_b200.topology import flatten
    g = Golden("insulin")
    rng = np.random.default_rng(8)
    sizes = [1, 255, 256, 257, 700, 2047, 2048, 2049, 2305]
    one = (g["xyz"], g["q"], g["r"], g["eps"], flatten(g.topology()))
    systems = [(rng.uniform(0, 10 + n ** (1 / 3) * 3, (n, 3)), rng.choice([-0.3, 0.3], n), np.full(n, 1.6),
                np.full(n, 0.1), None) for n in sizes] + [one] * 45
    b = DeviceBatch(systems)
    assert b.natoms <= 16 * b.nsys ** 2
    terms = b.energy_terms()
    for s in range(len(sizes) + 1):
        assert torch.equal(DeviceBatch([systems[s]]).energy_terms()[0], terms[s]), s
    assert torch.equal(terms[-1], terms[len(sizes)])


@pytest.mark.parametrize("copies", [1, 10])
def test_nl_rows_past_the_stage(oracle, copies):
    """Rows of more candidates than the stage holds, listed in 2 to 5 groups of 32
    chunks, with one atom per warp and with two (24,000 atoms and more): half
    rows equal to the oracle's, order included, full rows in their order."""
    from protein_physics_b200.device import DeviceBatch
    x = np.random.default_rng(21).uniform(0, 17, (2600, 3))
    b = DeviceBatch([(x, np.zeros(len(x)), np.full(len(x), 1.9), np.full(len(x), 0.1), None)] * copies)
    assert (b.natoms >= 24000) == (copies == 10)
    b.build_nl()
    ptr, ocols = oracle.nl_build(x)
    for s in {0, copies - 1}:
        rp, cols, _ = b.nl_host(s, half=True)
        assert np.array_equal(rp, ptr) and np.array_equal(cols, ocols), s
        frp, fcols, _ = b.nl_host(s, half=False)
        J = np.repeat(np.arange(len(x)), np.diff(frp))
        assert np.diff(frp).max() > 1536 and len(fcols) == 2 * len(ocols)
        assert np.array_equal(fcols[fcols > J], ocols), s
        srp, scols, _ = b.nl_host(s, half=False, short=True)
        r2 = ((x[J] - x[fcols]) ** 2).sum(1)
        reach = 2 * 1.9 + 2 * b.params.probe_r + 2 * np.sqrt(b.params.half_skin2) + 1e-6
        assert np.array_equal(scols, fcols[r2 < reach * reach]), s
