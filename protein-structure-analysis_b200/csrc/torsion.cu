// Torsion-space kinematics and the gradient-guided (MALA) torsion sampler.
//
// The sampler's coordinates are the rotatable-bond torsions: rotating bond
// k by θ turns its j-side about the axis x_i -> x_j (the reference's move,
// rodrigues physics_engine.cpp:1848-1862).  On a tree the j-sides are
// nested or disjoint (AlmaTorsionTree), which gives
//
//   gradient  dE/dθ_k = u_k · Σ_{m in side k} (x_m - x_i) × ∇_m E, from one
//             prefix sum by tiles of atoms of ((x_m - c) × ∇_m E, ∇_m E)
//             (a j-side is a range plus a few explicit atoms);
//   apply     all bonds at once: with every axis taken from the current
//             coordinates, turning the innermost bonds first equals the
//             reference's one-after-the-other moves with updated axes, so
//             atom m moves by T_k = A_root ∘ ... ∘ A_parent ∘ A_k, k = the
//             innermost bond holding m.  T is built per bond by pointer
//             jumping (log2(depth) rounds) inside one cluster per system;
//   MALA      θ' = θ + clip(-½ σ² β ∇_θE, ±c σ) + σ ξ per bond (σ_k =
//             state scale × step × lever scale), accepted with the
//             Metropolis–Hastings ratio of the Langevin proposal densities;
//             Philox draws keyed by (seed, system, step, bond).
#include <cooperative_groups.h>

#include <algorithm>

#include "alma_common.cuh"

namespace alma {

namespace cg = cooperative_groups;

struct Affine {
    double m[12];  // row-major 3x3 rotation, then translation
};

__device__ __forceinline__ Affine affine_compose(const Affine &A, const Affine &B) {  // A ∘ B
    Affine C;
#pragma unroll
    for (int r = 0; r < 3; ++r) {
#pragma unroll
        for (int c = 0; c < 3; ++c)
            C.m[3 * r + c] = A.m[3 * r] * B.m[c] + A.m[3 * r + 1] * B.m[3 + c] + A.m[3 * r + 2] * B.m[6 + c];
        C.m[9 + r] = A.m[3 * r] * B.m[9] + A.m[3 * r + 1] * B.m[10] + A.m[3 * r + 2] * B.m[11] + A.m[9 + r];
    }
    return C;
}

__device__ __forceinline__ void affine_load(Affine &A, const double *p) {
#pragma unroll
    for (int q = 0; q < 12; ++q) A.m[q] = p[q];
}

__device__ __forceinline__ void affine_store(const Affine &A, double *p) {
#pragma unroll
    for (int q = 0; q < 12; ++q) p[q] = A.m[q];
}

// Rotation by angle d about the unit axis through o along (pj - pi).
__device__ __forceinline__ Affine bond_rotation(double4 pi, double4 pj, double d) {
    Affine A;
    double ux = pj.x - pi.x, uy = pj.y - pi.y, uz = pj.z - pi.z;
    const double l = sqrt(ux * ux + uy * uy + uz * uz);
    if (d == 0.0 || l < 1e-10) {
        for (int q = 0; q < 12; ++q) A.m[q] = 0.0;
        A.m[0] = A.m[4] = A.m[8] = 1.0;
        return A;
    }
    ux /= l; uy /= l; uz /= l;
    const double c = cos(d), s = sin(d), k = 1.0 - c;
    A.m[0] = c + ux * ux * k;      A.m[1] = ux * uy * k - uz * s; A.m[2] = ux * uz * k + uy * s;
    A.m[3] = uy * ux * k + uz * s; A.m[4] = c + uy * uy * k;      A.m[5] = uy * uz * k - ux * s;
    A.m[6] = uz * ux * k - uy * s; A.m[7] = uz * uy * k + ux * s; A.m[8] = c + uz * uz * k;
    A.m[9] = pi.x - (A.m[0] * pi.x + A.m[1] * pi.y + A.m[2] * pi.z);
    A.m[10] = pi.y - (A.m[3] * pi.x + A.m[4] * pi.y + A.m[5] * pi.z);
    A.m[11] = pi.z - (A.m[6] * pi.x + A.m[7] * pi.y + A.m[8] * pi.z);
    return A;
}

// Turns every bond of a system at once: T_k for every bond (pointer jumping),
// then the atoms.  One cluster of CL CTAs per system; CTA r holds the bonds
// [r per, (r + 1) per) in its shared memory (transforms by component, so a
// warp's own reads are free of conflicts) and reads parents through
// distributed shared memory: a round is one such read and a cluster barrier,
// where the L2 round trips of a global buffer made it 7 us.  A system with
// more bonds than the cluster holds works in the global buffers instead.
// One system of 16k atoms and 4,000 bonds: 468 us with one CTA, 85 us as a
// cluster on global buffers, 31 us here.  The compositions and their order
// depend on neither CL nor the buffer.
constexpr int COMPOSE_THREADS = 512;
constexpr int COMPOSE_HOLD = 1024;  // bonds per CTA: 2 x 12 doubles each, 200 KB
constexpr size_t COMPOSE_SMEM = (size_t)COMPOSE_HOLD * 2 * (12 * sizeof(double) + sizeof(int32_t));

// Where the transforms and parents live: shared memory of the cluster, or
// global buffers.  Buffer 0 / 1 alternate between rounds.
template <int CL>
struct SharedBonds {
    double *T;    // [2][12][COMPOSE_HOLD]
    int32_t *P;   // [2][COMPOSE_HOLD]
    int per;
    __device__ __forceinline__ const double *peer(int buf, int rank) const {
        double *q = T + (size_t)buf * 12 * COMPOSE_HOLD;
        if constexpr (CL > 1) q = cg::this_cluster().map_shared_rank(q, rank);
        return q;
    }
    __device__ __forceinline__ void load(Affine &A, int buf, int k) const {
        const double *q = peer(buf, k / per) + k % per;
#pragma unroll
        for (int d = 0; d < 12; ++d) A.m[d] = q[d * COMPOSE_HOLD];
    }
    __device__ __forceinline__ void store(const Affine &A, int buf, int k) const {  // own bonds only
        double *q = T + (size_t)buf * 12 * COMPOSE_HOLD + k % per;
#pragma unroll
        for (int d = 0; d < 12; ++d) q[d * COMPOSE_HOLD] = A.m[d];
    }
    __device__ __forceinline__ int parent(int buf, int k) const {
        int32_t *q = P + buf * COMPOSE_HOLD;
        if constexpr (CL > 1) q = cg::this_cluster().map_shared_rank(q, k / per);
        return q[k % per];
    }
    __device__ __forceinline__ void set_parent(int buf, int k, int p) const { P[buf * COMPOSE_HOLD + k % per] = p; }
};

struct GlobalBonds {
    double *T[2];
    int32_t *P[2];
    __device__ __forceinline__ void load(Affine &A, int buf, int k) const { affine_load(A, T[buf] + 12 * (size_t)k); }
    __device__ __forceinline__ void store(const Affine &A, int buf, int k) const {
        affine_store(A, T[buf] + 12 * (size_t)k);
    }
    __device__ __forceinline__ int parent(int buf, int k) const { return P[buf][k]; }
    __device__ __forceinline__ void set_parent(int buf, int k, int p) const { P[buf][k] = p; }
};

// Bonds [k0, k1) of the system are this CTA's; every CTA of the cluster takes
// part in every barrier.
template <int CL, typename Bonds>
__device__ __forceinline__ void apply_torsions(const Bonds &B, int (*any_of)[8], int rank, int k0, int k1, int r0,
                                               int a0, int a1, double *xyz, const AlmaTopo &t,
                                               const int32_t *rb_parent, const int32_t *atom_rb, const double *delta) {
    auto sync = [] {
        if constexpr (CL > 1) cg::this_cluster().sync();
        else __syncthreads();
    };
    for (int k = k0 + (int)threadIdx.x; k < k1; k += COMPOSE_THREADS) {
        const int g = r0 + k;
        B.store(bond_rotation(ld_xyz(xyz, t.rb_ij[2 * g]), ld_xyz(xyz, t.rb_ij[2 * g + 1]), delta[g]), 0, k);
        B.set_parent(0, k, rb_parent[g]);
    }
    sync();
    int cur = 0;
    for (int round = 0; round < 32; ++round) {
        bool any = false;
        for (int k = k0 + (int)threadIdx.x; k < k1; k += COMPOSE_THREADS) {
            const int p = B.parent(cur, k);
            Affine Tk;
            B.load(Tk, cur, k);
            if (p >= 0) {
                Affine Tp;
                B.load(Tp, cur, p);
                B.set_parent(cur ^ 1, k, B.parent(cur, p));
                Tk = affine_compose(Tp, Tk);
                any = true;
            } else {
                B.set_parent(cur ^ 1, k, -1);
            }
            B.store(Tk, cur ^ 1, k);
        }
        cur ^= 1;
        const int mine = __syncthreads_or(any);
        if constexpr (CL > 1) {
            // every CTA tells every other; a slot is written again two rounds
            // on, behind another cluster barrier
            if (threadIdx.x < CL) cg::this_cluster().map_shared_rank(&any_of[round & 1][0], threadIdx.x)[rank] = mine;
            cg::this_cluster().sync();
            int all = 0;
#pragma unroll
            for (int r = 0; r < CL; ++r) all |= any_of[round & 1][r];
            if (!all) break;
        } else if (!mine) {
            break;
        }
    }
    // the transforms are complete and every axis has been read
    for (int m = a0 + rank * COMPOSE_THREADS + (int)threadIdx.x; m < a1; m += CL * COMPOSE_THREADS) {
        const int k = atom_rb[m];
        if (k < 0) continue;
        Affine A;
        B.load(A, cur, k);
        double4 p = ld_xyz(xyz, m);
        const double x = p.x, y = p.y, z = p.z;
        p.x = A.m[0] * x + A.m[1] * y + A.m[2] * z + A.m[9];
        p.y = A.m[3] * x + A.m[4] * y + A.m[5] * z + A.m[10];
        p.z = A.m[6] * x + A.m[7] * y + A.m[8] * z + A.m[11];
        *reinterpret_cast<double4 *>(xyz + 4 * (size_t)m) = p;
    }
    sync();  // no CTA leaves while another may still read its shared memory
}

struct ApplyArgs {
    const int32_t *atom_off;
    double *xyz;
    AlmaTopo t;
    const int32_t *rb_parent, *atom_rb;
    const double *delta;
    const uint8_t *mask;
    double *Tbuf;
    int32_t *Pbuf;
};

template <int CL>
__device__ __forceinline__ void apply_system(const ApplyArgs &A, int s) {
    extern __shared__ double compose_smem[];
    __shared__ int any_of[2][8];  // per round parity and CTA of the cluster: bonds still climbing
    const int rank = CL > 1 ? (int)cg::this_cluster().block_rank() : 0;
    const int r0 = A.t.rb_off[s], nr = A.t.rb_off[s + 1] - r0;
    const int per = max(1, (nr + CL - 1) / CL);
    const int k0 = min(nr, rank * per), k1 = min(nr, k0 + per);
    const int a0 = A.atom_off[s], a1 = A.atom_off[s + 1];
    if (per <= COMPOSE_HOLD) {
        const SharedBonds<CL> B{compose_smem, reinterpret_cast<int32_t *>(compose_smem + 24 * COMPOSE_HOLD), per};
        apply_torsions<CL>(B, any_of, rank, k0, k1, r0, a0, a1, A.xyz, A.t, A.rb_parent, A.atom_rb, A.delta);
    } else {
        const size_t n = (size_t)A.t.nrb;
        const GlobalBonds B{{A.Tbuf + 12 * (size_t)r0, A.Tbuf + 12 * (n + r0)}, {A.Pbuf + r0, A.Pbuf + n + r0}};
        apply_torsions<CL>(B, any_of, rank, k0, k1, r0, a0, a1, A.xyz, A.t, A.rb_parent, A.atom_rb, A.delta);
    }
}

template <int CL>
__global__ void __launch_bounds__(COMPOSE_THREADS) torsion_apply_kernel(ApplyArgs A, int limit) {
    const int s = blockIdx.x / CL;
    if (A.mask && !A.mask[s]) return;                          // the whole cluster
    if (A.t.rb_off[s + 1] - A.t.rb_off[s] > limit) return;  // likewise
    apply_system<CL>(A, s);
}

// An uneven batch: the host knows the number of systems and of bonds, not the
// sizes, and shapes the clusters for the mean.  Systems of more bonds than
// such a cluster holds (`limit`) are left to this kernel, a few clusters of 8 CTAs
// that find them 512 systems at a time and share them out in order.  A batch
// without any pays 4-5 us.  4,030 residues among 99 chains of 64: 2,761 us on
// the one CTA of the mean (2,132 as one CTA of twice the threads, atoms apart),
// 435 here; 1,000 among 40 of 64: 618 and 50.
constexpr int LARGE_CTAS = 8, LARGE_CLUSTERS = 15;  // as many as fit at one CTA per SM

__global__ void __launch_bounds__(COMPOSE_THREADS) torsion_apply_large_kernel(ApplyArgs A, int nsys, int limit) {
    __shared__ unsigned found[COMPOSE_THREADS / 32];
    const int cluster = blockIdx.x / LARGE_CTAS, clusters = gridDim.x / LARGE_CTAS;
    int seen = 0;
    for (int s0 = 0; s0 < nsys; s0 += COMPOSE_THREADS) {
        const int s = s0 + (int)threadIdx.x;
        const bool large = s < nsys && (!A.mask || A.mask[s]) && A.t.rb_off[s + 1] - A.t.rb_off[s] > limit;
        const unsigned m = __ballot_sync(0xffffffffu, large);
        if ((threadIdx.x & 31) == 0) found[threadIdx.x >> 5] = m;
        if (!__syncthreads_or(large)) continue;
        for (int w = 0; w < COMPOSE_THREADS / 32; ++w)
            for (unsigned rest = found[w]; rest; rest &= rest - 1u)
                if (seen++ % clusters == cluster) apply_system<LARGE_CTAS>(A, s0 + 32 * w + __ffs(rest) - 1);
        __syncthreads();  // found[] is written again
    }
}

struct V6 {
    double v[6];
};

__device__ __forceinline__ V6 v6_add(const V6 &a, const V6 &b) {
    V6 c;
#pragma unroll
    for (int q = 0; q < 6; ++q) c.v[q] = a.v[q] + b.v[q];
    return c;
}

// Inclusive block scan of V6 (blockDim.x multiple of 32, <= 1024).
__device__ __forceinline__ V6 block_scan6(V6 x, V6 *sm, V6 &total) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        V6 y;
#pragma unroll
        for (int q = 0; q < 6; ++q) y.v[q] = __shfl_up_sync(0xffffffffu, x.v[q], o);
        if (lane >= o) x = v6_add(x, y);
    }
    if (lane == 31) sm[wid] = x;
    __syncthreads();
    if (wid == 0) {
        V6 w;
#pragma unroll
        for (int q = 0; q < 6; ++q) w.v[q] = lane < nw ? sm[lane].v[q] : 0.0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            V6 y;
#pragma unroll
            for (int q = 0; q < 6; ++q) y.v[q] = __shfl_up_sync(0xffffffffu, w.v[q], o);
            if (lane >= o) w = v6_add(w, y);
        }
        sm[lane] = w;  // inclusive warp-total prefix
    }
    __syncthreads();
    if (wid > 0) x = v6_add(x, sm[wid - 1]);
    total = sm[nw - 1];
    __syncthreads();
    return x;
}

// Torsion gradient.  A bond's sum runs over an atom range [lo, hi) plus a few
// explicit atoms; the range is prefix(hi) - prefix(lo), a prefix the sum of the
// tiles before the atom, tile after tile, plus its place in its own tile: the
// order in which one CTA scans a system.  The order is kept for the sake of the
// sampler, whose chains follow the last bit of the gradient (an extreme atom
// sits on a cell face of the list); tiles and bonds of all systems run at once
// instead (16k atoms, 4,000 bonds, one system: 372 -> 13 us in two launches).
constexpr int TG_TILE = 1024;

__device__ __forceinline__ V6 torque_of(const double *xyz, const double *grad, int m, double4 c) {
    const double4 p = ld_xyz(xyz, m), g = ld_xyz(grad, m);
    const double rx = p.x - c.x, ry = p.y - c.y, rz = p.z - c.z;
    V6 x;
    x.v[0] = ry * g.z - rz * g.y;
    x.v[1] = rz * g.x - rx * g.z;
    x.v[2] = rx * g.y - ry * g.x;
    x.v[3] = g.x; x.v[4] = g.y; x.v[5] = g.z;
    return x;
}

// Inclusive prefixes of ((x_m - c) × g_m, g_m) within each tile -> P[6 m], the
// tile's total -> tot[6 slot] (c: the system's first atom).
__global__ void __launch_bounds__(TG_TILE)
torsion_prefix_kernel(const int32_t *__restrict__ atom_off, int nsys, const double *__restrict__ xyz,
                      const double *__restrict__ grad, const uint8_t *__restrict__ mask, double *__restrict__ P,
                      double *__restrict__ tot) {
    __shared__ V6 sm[32];
    const int s = sys_of_tile<TG_TILE>(atom_off, nsys, blockIdx.x);
    if (mask && !mask[s]) return;
    const int a0 = atom_off[s], a1 = atom_off[s + 1];
    const int m0 = a0 + ((int)blockIdx.x - tile_base<TG_TILE>(atom_off, s)) * TG_TILE;
    if (m0 >= a1) return;
    const int m = m0 + (int)threadIdx.x;
    V6 x = {};
    if (m < a1) x = torque_of(xyz, grad, m, ld_xyz(xyz, a0));
    V6 total;
    const V6 inc = block_scan6(x, sm, total);
    if (m < a1)
        for (int q = 0; q < 6; ++q) P[6 * (size_t)m + q] = inc.v[q];
    if (threadIdx.x == 0)
        for (int q = 0; q < 6; ++q) tot[6 * (size_t)blockIdx.x + q] = total.v[q];
}

// Eight lanes per bond: the torsion derivative from the prefixes.  A bond has
// few explicit atoms and a serial tail (a root, three quotients), so a warp per
// bond left most lanes idle and batches of many chains queued for it (400
// chains of 64 residues, 102k bonds: 87 -> 37 us).  The explicit atoms are summed
// as a warp would: atom e in the share of lane e mod 32, the shares by halves.
constexpr int TG_LANES = 8;

__global__ void __launch_bounds__(256)
torsion_grad_kernel(const int32_t *__restrict__ atom_off, int nsys, const double *__restrict__ xyz,
                    const double *__restrict__ grad, AlmaTopo t, const uint8_t *__restrict__ mask,
                    const double *__restrict__ P, const double *__restrict__ tot, double *__restrict__ gtheta) {
    const int k = (int)((blockIdx.x * blockDim.x + threadIdx.x) / TG_LANES), lane = threadIdx.x % TG_LANES;
    const unsigned group = 0xffu << (threadIdx.x & 24u);  // the lanes of this bond
    if (k >= t.nrb) return;
    const int s = sys_of_atom(t.rb_off, nsys, k);
    if (mask && !mask[s]) return;
    const int a0 = atom_off[s];
    if (atom_off[s + 1] <= a0) return;
    const double4 c = ld_xyz(xyz, a0);
    const int64_t e0 = t.side_ptr[k], e1 = t.side_ptr[k + 1];
    auto share = [&](int u) {
        V6 x = {};
        for (int64_t e = e0 + TG_LANES * u + lane; e < e1; e += 32) x = v6_add(x, torque_of(xyz, grad, t.side_idx[e], c));
        return x;
    };
    V6 S = share(0);
    if (e1 - e0 > TG_LANES) {
        S = v6_add(S, share(2));
        V6 x = share(1);
        x = v6_add(x, share(3));
        S = v6_add(S, x);
    }
    __syncwarp(group);
#pragma unroll
    for (int q = 0; q < 6; ++q)
#pragma unroll
        for (int o = TG_LANES / 2; o > 0; o >>= 1) S.v[q] += __shfl_xor_sync(group, S.v[q], o);
    const int lo = t.side_lo[k], hi = t.side_hi[k];
    if (hi > lo) {
        // lane q < 6: component q of the range
        const int a1 = atom_off[s + 1], q = lane < 6 ? lane : 0;
        const double *ts = tot + 6 * (size_t)tile_base<TG_TILE>(atom_off, s) + q;
        const int tl = (lo - a0) / TG_TILE, th = hi < a1 ? (hi - a0) / TG_TILE : (a1 - a0 - 1) / TG_TILE + 1;
        double carry = 0.0, before = 0.0;
#pragma unroll 8
        for (int u = 0; u < th; ++u) {
            if (u == tl) before = carry;
            carry += ts[6 * (size_t)u];
        }
        if (th == tl) before = carry;
        auto pick = [&](const V6 &x) {
            double r = x.v[0];
#pragma unroll
            for (int d = 1; d < 6; ++d) r = q == d ? x.v[d] : r;
            return r;
        };
        double ph = carry;
        if (hi < a1) ph = carry + P[6 * (size_t)hi + q] - pick(torque_of(xyz, grad, hi, c));
        const double pl = before + P[6 * (size_t)lo + q] - pick(torque_of(xyz, grad, lo, c));
        const double sum = pick(S) + (ph - pl);
#pragma unroll
        for (int d = 0; d < 6; ++d) S.v[d] = __shfl_sync(group, sum, d, TG_LANES);
    }
    if (lane == 0) {
        const double4 pi = ld_xyz(xyz, t.rb_ij[2 * k]), pj = ld_xyz(xyz, t.rb_ij[2 * k + 1]);
        double ux = pj.x - pi.x, uy = pj.y - pi.y, uz = pj.z - pi.z;
        const double l = sqrt(ux * ux + uy * uy + uz * uz);
        double gk = 0.0;
        if (l >= 1e-10) {
            ux /= l; uy /= l; uz /= l;
            const double ox = pi.x - c.x, oy = pi.y - c.y, oz = pi.z - c.z;
            // Σ (x - o) × g = Σ (x - c) × g - (o - c) × Σ g
            const double tx = S.v[0] - (oy * S.v[5] - oz * S.v[4]);
            const double ty = S.v[1] - (oz * S.v[3] - ox * S.v[5]);
            const double tz = S.v[2] - (ox * S.v[4] - oy * S.v[3]);
            gk = ux * tx + uy * ty + uz * tz;
        }
        gtheta[k] = gk;
    }
}

// ---- MALA ------------------------------------------------------------------
__device__ __forceinline__ int sys_of_bond(const int32_t *rb_off, int nsys, int k) {
    return sys_of_atom(rb_off, nsys, k);  // same search over the [nsys+1] offsets
}

__device__ __forceinline__ void mala_key(uint64_t seed, int s, uint32_t &k0, uint32_t &k1) {
    k0 = (uint32_t)seed ^ (0x85EBCA6Bu * (uint32_t)(s + 1));
    k1 = (uint32_t)(seed >> 32) ^ 0x27D4EB2Fu;
}

// Truncated Langevin drift of bond k (MALTA: Roberts & Tweedie, Bernoulli
// 2:341, 1996): -½ σ² β g clipped to ±clip·σ.  Steep clashes give
// gradients of 1e3-1e6 kcal/mol/rad whose untruncated drift would throw
// the proposal far away; any deterministic drift keeps detailed balance as
// long as the same function enters the forward and reverse densities.
__device__ __forceinline__ double mala_drift(double sg, double beta, double g, double clip) {
    const double mu = -0.5 * sg * sg * beta * g, lim = clip * sg;
    return fmin(fmax(mu, -lim), lim);
}

__global__ void mala_propose_kernel(int nrb, int nsys, const int32_t *__restrict__ rb_off,
                                    const double *__restrict__ gtheta, const double *__restrict__ sigma,
                                    const AlmaMalaState *__restrict__ st, AlmaMalaConfig cfg,
                                    const uint8_t *__restrict__ mask, double *__restrict__ delta) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nrb) return;
    const int s = sys_of_bond(rb_off, nsys, k);
    if (mask && !mask[s]) return;
    const double sg = sigma[k] * st[s].scale;
    if (!(sg > 0.0)) {
        delta[k] = 0.0;
        return;
    }
    const int kl = k - rb_off[s];
    const uint64_t step = (uint64_t)st[s].step;
    uint32_t k0, k1;
    mala_key(cfg.seed, s, k0, k1);
    const Philox4 r = philox4x32_10((uint32_t)step, (uint32_t)(step >> 32), (uint32_t)s,
                                    0x40000000u + ((uint32_t)kl >> 1), k0, k1);
    // Box–Muller: two normals per draw, bond parity picks one
    const double u1 = 1.0 - u01_from(r.v[0], r.v[1]), u2 = u01_from(r.v[2], r.v[3]);
    const double rad = sqrt(-2.0 * log(u1));
    const double xi = (kl & 1) ? rad * sin(6.283185307179586 * u2) : rad * cos(6.283185307179586 * u2);
    delta[k] = mala_drift(sg, st[s].beta, gtheta[k], cfg.drift_clip) + sg * xi;
}

// One CTA per system: Metropolis–Hastings test of the Langevin proposal,
// then the step-scale adaptation window.  1,024 threads: a bond costs three
// FP64 divisions behind its loads, and 4,000 bonds on 256 threads took 17 us (now 6).
constexpr int ACCEPT_THREADS = 1024;

__global__ void __launch_bounds__(ACCEPT_THREADS) mala_accept_kernel(int nsys, const int32_t *__restrict__ rb_off, const double *__restrict__ delta,
                                   const double *__restrict__ g_old, const double *__restrict__ g_new,
                                   const double *__restrict__ sigma, const double *__restrict__ terms_new,
                                   AlmaMalaConfig cfg, const uint8_t *__restrict__ mask,
                                   AlmaMalaState *__restrict__ st, uint8_t *__restrict__ accept) {
    __shared__ double sm[32];
    const int s = blockIdx.x;
    if (mask && !mask[s]) return;
    const double beta = st[s].beta, scale = st[s].scale;
    double fwd = 0.0, rev = 0.0;
    for (int k = rb_off[s] + threadIdx.x; k < rb_off[s + 1]; k += blockDim.x) {
        const double sg = sigma[k] * scale;
        if (!(sg > 0.0)) continue;
        const double rf = delta[k] - mala_drift(sg, beta, g_old[k], cfg.drift_clip);
        const double rr = -delta[k] - mala_drift(sg, beta, g_new[k], cfg.drift_clip);
        fwd += rf * rf / (2.0 * sg * sg);
        rev += rr * rr / (2.0 * sg * sg);
    }
    fwd = block_sum(fwd, sm);
    rev = block_sum(rev, sm);
    if (threadIdx.x == 0) {
        AlmaMalaState S = st[s];
        const double En = terms_new[5 * (size_t)s + 4];
        const double log_alpha = -beta * (En - S.energy) - rev + fwd;
        uint32_t k0, k1;
        mala_key(cfg.seed, s, k0, k1);
        const Philox4 r = philox4x32_10((uint32_t)S.step, (uint32_t)(S.step >> 32), (uint32_t)s, 0x3FFFFFFFu, k0, k1);
        const double u = u01_from(r.v[0], r.v[1]);
        const int acc = isfinite(En) && isfinite(log_alpha) && (log_alpha >= 0.0 || log(u) < log_alpha);
        accept[s] = (uint8_t)acc;
        S.log_alpha = log_alpha;
        S.n_proposed++;
        if (acc) {
            S.energy = En;
            S.n_accepted++;
        }
        S.acc_win += acc;
        if (cfg.tune_freq > 0 && ++S.tot_win == cfg.tune_freq) {
            const double rate = (double)S.acc_win / (double)cfg.tune_freq;
            if (rate > cfg.target_hi) S.scale = fmin(cfg.scale_max, S.scale * cfg.scale_up);
            else if (rate < cfg.target_lo) S.scale = fmax(cfg.scale_min, S.scale * cfg.scale_down);
            S.acc_win = 0;
            S.tot_win = 0;
        }
        S.step++;
        st[s] = S;
    }
}

// Rejected systems take back their saved coordinates and Born radii;
// accepted systems take the proposal's torsion gradient.
__global__ void mala_select_kernel(int natoms, int nrb, int nsys, const int32_t *__restrict__ atom_off,
                                   const int32_t *__restrict__ rb_off, const uint8_t *__restrict__ accept,
                                   const uint8_t *__restrict__ mask, const double *__restrict__ xyz_old,
                                   const double *__restrict__ born_old, double *__restrict__ xyz,
                                   double *__restrict__ born, const double *__restrict__ g_new,
                                   double *__restrict__ g_cur) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q < natoms) {
        const int s = sys_of_atom(atom_off, nsys, q);
        if ((!mask || mask[s]) && !accept[s]) {
            *reinterpret_cast<double4 *>(xyz + 4 * (size_t)q) = ld_xyz(xyz_old, q);
            born[q] = born_old[q];
        }
    }
    if (q < nrb && g_new && g_cur) {
        const int s = sys_of_bond(rb_off, nsys, q);
        if ((!mask || mask[s]) && accept[s]) g_cur[q] = g_new[q];
    }
}

static size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

}  // namespace alma

using namespace alma;

extern "C" size_t alma_torsion_workspace_bytes(int32_t natoms, int32_t nsys, int32_t nrb) {
    const size_t n = natoms > 0 ? (size_t)natoms : 0, S = nsys > 0 ? (size_t)nsys : 0, r = nrb > 0 ? (size_t)nrb : 0;
    const size_t compose = align256(sizeof(double) * 24 * r) + align256(sizeof(int32_t) * 2 * r);
    const size_t prefix = align256(sizeof(double) * 6 * n) + align256(sizeof(double) * 6 * (n / TG_TILE + S));
    return std::max(compose, prefix) + 256;
}

static int torsion_args(const AlmaBatch *b, const AlmaTopo *t, const char *who) {
    if (!b || !t || b->nsys <= 0 || b->natoms < 0 || !b->atom_off || !b->xyz)
        return alma_set_error(ALMA_EINVAL, "%s: bad arguments", who);
    if (t->nrb > 0 && (!t->rb_off || !t->rb_ij || !t->side_ptr || !t->side_lo || !t->side_hi))
        return alma_set_error(ALMA_EINVAL, "%s: topology without rotatable-bond arrays", who);
    if (!t->rb_off) return alma_set_error(ALMA_EINVAL, "%s: topology without rb_off", who);
    return ALMA_OK;
}

extern "C" int alma_torsion_grad(const AlmaBatch *b, const AlmaTopo *t, const double *grad, const uint8_t *sys_mask,
                                 void *workspace, double *gtheta, void *stream) {
    int rc = torsion_args(b, t, "alma_torsion_grad");
    if (rc) return rc;
    if (!grad || !gtheta || !workspace) return alma_set_error(ALMA_EINVAL, "alma_torsion_grad: null buffer");
    if (b->natoms == 0 || t->nrb == 0) return ALMA_OK;
    cudaStream_t st = (cudaStream_t)stream;
    double *P = (double *)workspace;
    double *tot = (double *)((char *)workspace + align256(sizeof(double) * 6 * (size_t)b->natoms));
    torsion_prefix_kernel<<<tile_slots<TG_TILE>(b->natoms, b->nsys), TG_TILE, 0, st>>>(b->atom_off, b->nsys, b->xyz,
                                                                                      grad, sys_mask, P, tot);
    const int per_block = 256 / TG_LANES;
    torsion_grad_kernel<<<(t->nrb + per_block - 1) / per_block, 256, 0, st>>>(b->atom_off, b->nsys, b->xyz, grad, *t,
                                                                              sys_mask, P, tot, gtheta);
    ALMA_LAUNCH_CHECK_N("alma_torsion_grad", 2);
    return ALMA_OK;
}

extern "C" int alma_torsion_apply(const AlmaBatch *b, const AlmaTopo *t, const AlmaTorsionTree *tree,
                                  const double *delta, const uint8_t *sys_mask, void *workspace, void *stream) {
    int rc = torsion_args(b, t, "alma_torsion_apply");
    if (rc) return rc;
    if (!tree || !tree->rb_parent || !tree->atom_rb || !delta || !workspace)
        return alma_set_error(ALMA_EINVAL, "alma_torsion_apply: null buffer");
    if (b->natoms == 0 || t->nrb == 0) return ALMA_OK;
    cudaStream_t st = (cudaStream_t)stream;
    double *Tbuf = (double *)workspace;
    int32_t *Pbuf = (int32_t *)((char *)workspace + align256(sizeof(double) * 24 * (size_t)t->nrb));
    // About one bond per thread of the mean system, up to 8 CTAs (the portable
    // cluster): past that a wider cluster only adds barrier time.
    const int avg = t->nrb / b->nsys;
    const int cl = avg <= COMPOSE_THREADS ? 1 : avg <= 2 * COMPOSE_THREADS ? 2 : avg <= 4 * COMPOSE_THREADS ? 4 : 8;
    const ApplyArgs A{b->atom_off, b->xyz, *t, tree->rb_parent, tree->atom_rb, delta, sys_mask, Tbuf, Pbuf};
    auto launch = [&](auto kfn, int grid, int ctas, auto... args) {
        const cudaError_t e = cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)COMPOSE_SMEM);
        if (e != cudaSuccess) return e;
        return alma_launch_cluster(kfn, (unsigned)grid, COMPOSE_THREADS, (unsigned)ctas, COMPOSE_SMEM, st, A, args...);
    };
    const int limit = cl * COMPOSE_HOLD;
    const bool large = b->nsys > 1 && cl < LARGE_CTAS && t->nrb > limit;  // there may be one
    ALMA_CUDA_TRY(launch(cl == 1 ? torsion_apply_kernel<1> : cl == 2 ? torsion_apply_kernel<2>
                         : cl == 4 ? torsion_apply_kernel<4> : torsion_apply_kernel<8>,
                         b->nsys * cl, cl, large ? limit : 0x7fffffff));
    if (large)
        ALMA_CUDA_TRY(launch(torsion_apply_large_kernel, std::min(b->nsys, LARGE_CLUSTERS) * LARGE_CTAS, LARGE_CTAS,
                             b->nsys, limit));
    ALMA_LAUNCH_CHECK_N("alma_torsion_apply", large ? 2 : 1);
    return ALMA_OK;
}

extern "C" int alma_mala_propose(const AlmaTopo *t, int32_t nsys, const double *gtheta, const double *sigma,
                                 const AlmaMalaConfig *cfg, const AlmaMalaState *states, const uint8_t *sys_mask,
                                 double *delta, void *stream) {
    if (!t || nsys <= 0 || !t->rb_off || !gtheta || !sigma || !cfg || !states || !delta)
        return alma_set_error(ALMA_EINVAL, "alma_mala_propose: bad arguments");
    if (t->nrb == 0) return ALMA_OK;
    mala_propose_kernel<<<(t->nrb + 255) / 256, 256, 0, (cudaStream_t)stream>>>(t->nrb, nsys, t->rb_off, gtheta,
                                                                                sigma, states, *cfg, sys_mask, delta);
    ALMA_LAUNCH_CHECK("alma_mala_propose");
    return ALMA_OK;
}

extern "C" int alma_mala_accept(const AlmaTopo *t, int32_t nsys, const double *delta, const double *g_old,
                                const double *g_new, const double *sigma, const double *terms_new,
                                const AlmaMalaConfig *cfg, const uint8_t *sys_mask, AlmaMalaState *states,
                                uint8_t *accept, void *stream) {
    if (!t || nsys <= 0 || !t->rb_off || !delta || !g_old || !g_new || !sigma || !terms_new || !cfg || !states ||
        !accept)
        return alma_set_error(ALMA_EINVAL, "alma_mala_accept: bad arguments");
    mala_accept_kernel<<<nsys, ACCEPT_THREADS, 0, (cudaStream_t)stream>>>(nsys, t->rb_off, delta, g_old, g_new, sigma, terms_new,
                                                               *cfg, sys_mask, states, accept);
    ALMA_LAUNCH_CHECK("alma_mala_accept");
    return ALMA_OK;
}

extern "C" int alma_mala_select(AlmaBatch *b, const AlmaTopo *t, const uint8_t *accept, const uint8_t *sys_mask,
                                const double *xyz_old, const double *born_old, const double *g_new, double *g_cur,
                                void *stream) {
    if (!b || !t || !t->rb_off || !accept || !xyz_old || !born_old || !b->xyz || !b->born)
        return alma_set_error(ALMA_EINVAL, "alma_mala_select: bad arguments");
    const int n = std::max(b->natoms, t->nrb);
    if (n == 0) return ALMA_OK;
    mala_select_kernel<<<(n + 255) / 256, 256, 0, (cudaStream_t)stream>>>(b->natoms, t->nrb, b->nsys, b->atom_off,
                                                                          t->rb_off, accept, sys_mask, xyz_old,
                                                                          born_old, b->xyz, b->born, g_new, g_cur);
    ALMA_LAUNCH_CHECK("alma_mala_select");
    return ALMA_OK;
}
