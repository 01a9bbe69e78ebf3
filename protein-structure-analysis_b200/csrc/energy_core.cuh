// Per-atom cores of the energy evaluation (Born radius of one atom, pair
// energy and SASA of one half row, dihedral records), shared by the
// stand-alone kernels (energy.cu) and the rebuild inside the persistent MC
// kernel (mc.cu).
#pragma once
#include "alma_common.cuh"

namespace alma {

// (charge, R*, epsilon) in precision R.
template <typename R>
__device__ __forceinline__ void load_prm(const float *prm, const double *prm64, int i, R &q, R &rad, R &eps) {
    if constexpr (sizeof(R) == 4) {
        const float4 p = *reinterpret_cast<const float4 *>(prm + 4 * (size_t)i);
        q = p.x; rad = p.y; eps = p.z;
    } else {
        const double4 p = *reinterpret_cast<const double4 *>(prm64 + 4 * (size_t)i);
        q = p.x; rad = p.y; eps = p.z;
    }
}

// HCT Born radius of atom i over its full row (one warp; FP64 sum).  Issue and
// L1 wavefronts bound it (78 and 73 %), so an entry gathers its position in one
// load (WIDE) and the radius alone: 39 M entries at 65k atoms, 165 -> 159 us.
template <typename R, bool WIDE = false>
__device__ __forceinline__ void born_atom(int i, int lane, const double *__restrict__ xyz, const float *__restrict__ prm,
                                          const double *__restrict__ prm64, const int64_t *__restrict__ full_ptr,
                                          const int32_t *__restrict__ full_len, const uint32_t *__restrict__ full_cols,
                                          double *__restrict__ born) {
    R qi, ri, ei;
    load_prm<R>(prm, prm64, i, qi, ri, ei);
    const double4 pi = ld_xyz(xyz, i);
    double sum = 0.0;
    const int64_t end = full_ptr[i] + full_len[i];
    int64_t k = full_ptr[i] + lane;
    uint32_t nxt = k < end ? full_cols[k] : 0u;  // the next entry is fetched while this one is evaluated
    for (; k < end; k += 32) {
        const int j = (int)(nxt & ALMA_IDX_MASK);
        if (k + 32 < end) nxt = full_cols[k + 32];
        R rj;
        if constexpr (sizeof(R) == 4) rj = prm[4 * (size_t)j + 1];
        else rj = prm64[4 * (size_t)j + 1];
        const double r2d = d2_of(pi, ld_pos<WIDE>(xyz, j));
        const R r2 = (R)r2d;
        sum += (double)hct_term<R>(f_sqrt(r2), r2, ri, rj);
    }
    sum = warp_sum(sum);
    if (lane == 0) {
        const double r64 = prm64[4 * (size_t)i + 1];
        const double inv = 1.0 / r64 - 0.5 * sum;
        born[i] = 1.0 / fmax(inv, 2.0);
    }
}

// Per-warp buffers of the pair pass: entries that need more than the FP32
// pair terms wait here until 32 of them fill the warp's lanes (< 32 waiting +
// one chunk).
struct PairBuf {
    double sasa_r2[64];    // within SASA reach, in row order
    double near_r2[64];    // near pairs
    int32_t sasa_j[64], near_j[64];
};

// An FP32 reach or sigma (sum of radii, rounded) squared, widened past its
// rounding: what lies beyond cannot be within the FP64 one.
__device__ __forceinline__ float widened2(float d) { return d * d * 1.00001f; }

// Pair energy and SASA of atom i's half row (one warp): atom_e[2i] = pair
// sum of the row, atom_e[2i+1] = gamma * max(0, sa_i), also into sasa_out[i]
// when given.
//
// About one entry in ten is within SASA reach (an FP64 square root and
// division each) and one in thirty is near: a contact inside sigma (an FP64
// square root and two divisions) or a pair that GB's exponential reaches.  Done
// in place, some lane of nearly every chunk needs them and the whole warp
// waits.  Both are packed into `buf` and evaluated 32 at a time, so the loop
// itself is left with the far pairs; the values and the row order of the SASA
// recurrence are those of the entry-by-entry loop.  20 M half-row entries at 65k atoms:
// 223 -> 196 us.
template <typename R, bool WIDE = false>
__device__ __forceinline__ void pair_sasa_atom(const DevParams &P, int i, int lane, const double *__restrict__ xyz,
                                               const float *__restrict__ prm, const double *__restrict__ prm64,
                                               const double *__restrict__ born, const int64_t *__restrict__ half_ptr,
                                               const int32_t *__restrict__ half_len,
                                               const uint32_t *__restrict__ half_cols, int use_excl, PairBuf &buf,
                                               double *__restrict__ atom_e, double *__restrict__ sasa_out) {
    R qi, ri, ei;
    load_prm<R>(prm, prm64, i, qi, ri, ei);
    const R ai = (R)born[i];
    const double4 pi = ld_pos<WIDE>(xyz, i);
    const double ri64 = prm64[4 * (size_t)i + 1], ei64 = prm64[4 * (size_t)i + 2];
    const double rsi = ri64 + P.probe_r;
    const double cap_scale = 2.0 * 3.14159265358979323846 * rsi * rsi;
    const float reach_i = (float)(rsi + P.probe_r);
    double sa = 4.0 * 3.14159265358979323846 * rsi * rsi;
    double e = 0.0;
    int nsasa = 0, nnear = 0;
    const unsigned below = (1u << lane) - 1u;
    auto sasa = [&](int n) {
        double cap = 0.0;
        if (lane < n) {
            const double rsj = prm64[4 * (size_t)buf.sasa_j[lane] + 1] + P.probe_r;
            const double r = sqrt(buf.sasa_r2[lane]), dc = rsi + rsj;
            if (r < dc) cap = cap_scale * ((dc - r) / (2.0 * rsi));
        }
        sa = sasa_steps(sa, n, cap);
    };
    auto contacts = [&](int n) {
        if (lane >= n) return;
        const int j = buf.near_j[lane];
        const double4 q = *reinterpret_cast<const double4 *>(prm64 + 4 * (size_t)j);
        R qj, rj, ej;
        load_prm<R>(prm, prm64, j, qj, rj, ej);
        e += (double)pair_energy<R>(P, buf.near_r2[lane], qi * qj, ri + rj, ei * ej, ai, (R)born[j], ri64 + q.y,
                                    ei64 * q.z);
    };
    const int64_t beg = half_ptr[i], end = half_ptr[i] + half_len[i];
    // the next chunk's entry is fetched while this one is evaluated, and all
    // of an entry's gathers are issued together (one dependent round trip
    // per chunk; the 12-14 Å entries load parameters they do not use)
    uint32_t nxt = beg + lane < end ? half_cols[beg + lane] : 0u;
    for (int64_t k0 = beg; k0 < end; k0 += 32) {
        const int64_t k = k0 + lane;
        bool hit = false, near = false;
        int j = 0;
        double r2d = 0.0;
        if (k < end) {
            const uint32_t ent = nxt;
            if (k + 32 < end) nxt = half_cols[k + 32];
            j = (int)(ent & ALMA_IDX_MASK);
            const double4 pj = ld_pos<WIDE>(xyz, j);
            R qj, rj, ej;
            load_prm<R>(prm, prm64, j, qj, rj, ej);
            const R aj = (R)born[j];
            r2d = d2_of(pi, pj);
            const float r2 = (float)r2d;
            hit = r2 < widened2(reach_i + (float)rj);
            if (!(use_excl && (ent & ALMA_EXCL_BIT)) && r2d <= P.pair_cut2) {
                if constexpr (sizeof(R) == 4) {
                    const float sig = ri + rj;
                    near = r2 < fmaxf(widened2(sig), GB_FAR * (ai * aj));
                    if (!near) e += (double)pair_energy_far(P, r2, rsqrtf(r2), qi * qj, sig, ei * ej);
                } else {
                    e += (double)pair_energy<R>(P, r2d, qi * qj, ri + rj, ei * ej, ai, aj, 0.0, 0.0);
                }
            }
        }
        const unsigned mh = __ballot_sync(0xffffffffu, hit);
        if (hit) {
            const int at = nsasa + __popc(mh & below);
            buf.sasa_r2[at] = r2d;
            buf.sasa_j[at] = j;
        }
        nsasa += __popc(mh);
        if constexpr (sizeof(R) == 4) {
            const unsigned mn = __ballot_sync(0xffffffffu, near);
            if (near) {
                const int at = nnear + __popc(mn & below);
                buf.near_r2[at] = r2d;
                buf.near_j[at] = j;
            }
            nnear += __popc(mn);
        }
        if (nsasa >= 32) {
            __syncwarp();
            sasa(32);
            nsasa -= 32;
            double r2 = 0.0;
            int jj = 0;
            if (lane < nsasa) { r2 = buf.sasa_r2[32 + lane]; jj = buf.sasa_j[32 + lane]; }
            __syncwarp();
            if (lane < nsasa) { buf.sasa_r2[lane] = r2; buf.sasa_j[lane] = jj; }
            __syncwarp();
        }
        if constexpr (sizeof(R) == 4) {
            if (nnear >= 32) {
                __syncwarp();
                contacts(32);
                nnear -= 32;
                double r2 = 0.0;
                int jj = 0;
                if (lane < nnear) { r2 = buf.near_r2[32 + lane]; jj = buf.near_j[32 + lane]; }
                __syncwarp();
                if (lane < nnear) { buf.near_r2[lane] = r2; buf.near_j[lane] = jj; }
                __syncwarp();
            }
        }
    }
    __syncwarp();
    sasa(nsasa);
    if constexpr (sizeof(R) == 4) contacts(nnear);
    __syncwarp();  // the buffer is free for this warp's next atom
    e = warp_sum(e);
    if (lane == 0) {
        atom_e[2 * (size_t)i] = e;
        atom_e[2 * (size_t)i + 1] = P.gamma_sa * fmax(0.0, sa);
        if (sasa_out) sasa_out[i] = atom_e[2 * (size_t)i + 1];
    }
}

__device__ __forceinline__ double dihedral_angle(const double *xyz, int a, int b, int c, int d) {
    const double4 A = ld_xyz(xyz, a), B = ld_xyz(xyz, b), C = ld_xyz(xyz, c), D = ld_xyz(xyz, d);
    const double b1x = A.x - B.x, b1y = A.y - B.y, b1z = A.z - B.z;
    const double b2x = C.x - B.x, b2y = C.y - B.y, b2z = C.z - B.z;
    const double b3x = D.x - C.x, b3y = D.y - C.y, b3z = D.z - C.z;
    const double n1x = b1y * b2z - b1z * b2y, n1y = b1z * b2x - b1x * b2z, n1z = b1x * b2y - b1y * b2x;
    const double n2x = b2y * b3z - b2z * b3y, n2y = b2z * b3x - b2x * b3z, n2z = b2x * b3y - b2y * b3x;
    const double m1x = n1y * b2z - n1z * b2y, m1y = n1z * b2x - n1x * b2z, m1z = n1x * b2y - n1y * b2x;
    return atan2(m1x * n2x + m1y * n2y + m1z * n2z, n1x * n2x + n1y * n2y + n1z * n2z);
}

__device__ __forceinline__ double dih_record_energy(const double *xyz, const AlmaTopo &t, int r) {
    const int4 q = *reinterpret_cast<const int4 *>(t.dih_abcd + 4 * (size_t)r);
    const double phi = dihedral_angle(xyz, q.x, q.y, q.z, q.w);
    double E = 0.0;
    for (int k = t.term_off[r]; k < t.term_off[r + 1]; ++k)
        E += t.term_v2[k] * (1.0 + cos((double)t.term_n[k] * phi - t.term_gamma[k]));
    return E;
}

}  // namespace alma
