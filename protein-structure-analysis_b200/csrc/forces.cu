// Analytic gradient dE/dx of the full energy (the backward of alma_energy).
//
// E = Σ_pairs e(r_ij, a_i a_j) + E_SASA + E_dihedral + E_SS with the Born
// radii a_i = 1/max(1/rho_i - ½ Σ_j hct(r_ij; rho_i, rho_j), 2) (born_radii,
// physics_engine.cpp:2024-2039).  Three kernels:
//
//   pair   warp per atom over its FULL row: the direct pair force of every
//          non-excluded partner within 12 Å, gathered (each pair is seen
//          from both ends, so no atomics), and dE/da_i = Σ_j ∂e/∂(a_i a_j)·a_j,
//          kept as c_i = dE/da_i · a_i²/2 (0 where the radius is clamped);
//          the entries j > i within SASA reach are the SASA recurrence's, in
//          its order: sa <- sa - min(0.85 sa, cap_k) (:2068-2083), where an
//          entry that took the cap branch has the adjoint γ·π·R*·0.15^(number
//          of later entries that took the 0.85 branch); its force goes to both
//          atoms through 64-bit fixed-point atomics (integer adds: order
//          independent);
//   bonded thread per dihedral record / disulfide, fixed-point atomics.  The
//          reference angle is atan2(|b2| sinφ, cosφ) (its m1 = n1 × b2 is not
//          normalised, :1871-1887), and the gradient is that of this angle;
//   born   warp per atom over its FULL row: the chain rule through the
//          recomputed HCT integrals, Σ_j (c_i hct'(r; rho_i, rho_j) +
//          c_j hct'(r; rho_j, rho_i)) (x_i - x_j)/r, plus the pair and
//          fixed-point parts: the final gradient.
//
// Precision R: the pair and HCT derivative arithmetic (float in mixed mode;
// LJ and hard core inside sigma in FP64, as in the ΔE path), accumulation
// in FP64.  Every sum has a fixed order, so the gradient is deterministic.
#include "energy_core.cuh"

namespace alma {

constexpr double FIX_SCALE = 4294967296.0;  // 2^32: resolution 2.3e-10, range ±2.1e9
constexpr double FIX_INV = 1.0 / 4294967296.0;

__device__ __forceinline__ void fix_add(unsigned long long *slot, double v) {
    atomicAdd(slot, (unsigned long long)__double2ll_rn(v * FIX_SCALE));
}

// (dE/dr)/r of one pair and ∂E/∂(a_i a_j), pair_e (:2148-2164):
//   DH  K qq e^{-κr}/r            -> -e_dh (1/r + κ) / r
//   GB  C qq / f, f² = r² + A D, D = e^{-r²/4A}
//       -> -e_gb (2 - D/2) / (2 f²),   ∂/∂A = -e_gb D (1 + r²/4A) / (2 f²)
//   LJ  4√εε (s¹² - s⁶), s = σ/r  -> 4√εε (6 s⁶ - 12 s¹²) / r²
//   hard min(H x², cap), x = (rc/r)¹² - 1 -> -24 H x (rc/r)¹² / r² below the cap

// Debye-Hückel + GB: (dE/dr)/r, and ∂E/∂(a_i a_j) -> dEdA.
template <typename R>
__device__ __forceinline__ double grad_screened(const DevParams &P, R r2, R qp, R ai, R aj, double &dEdA) {
    R f_dh, f_gb;
    if constexpr (sizeof(R) == 4) {  // the fast FP32 forms of pair_energy (same error budget)
        const float rinv = rsqrtf(r2), r = r2 * rinv;
        const float kap = (float)P.kappa;
        const float edh = (float)P.coulomb_over_epsw * qp * rinv * __expf(-kap * r);
        f_dh = -edh * (rinv + kap) * rinv;
        const float A = ai * aj;
        const float r2_4A = 0.25f * __fdividef(r2, A);
        const float D = __expf(-r2_4A);
        const float f2 = r2 + A * D;
        const float rf2 = __fdividef(1.0f, f2);
        const float egb = (float)P.gb_coef * qp * rsqrtf(f2);
        f_gb = -egb * (2.0f - 0.5f * D) * 0.5f * rf2;
        dEdA = (double)(-egb * D * (1.0f + r2_4A) * 0.5f * rf2);
    } else {
        const R r = m_sqrt(r2);
        const R kap = (R)P.kappa;
        const R edh = (R)P.coulomb_over_epsw * qp / r * m_exp(-kap * r);
        f_dh = -edh * ((R)1 / r + kap) / r;
        const R A = ai * aj;
        const R D = m_exp(-r2 / ((R)4 * A));
        const R f2 = r2 + A * D;
        const R egb = (R)P.gb_coef * qp / m_sqrt(f2);
        f_gb = -egb * ((R)2 - (R)0.5 * D) / ((R)2 * f2);
        dEdA = (double)(-egb * D * ((R)1 + r2 / ((R)4 * A)) / ((R)2 * f2));
    }
    return (double)f_dh + (double)f_gb;
}

// The same of a far pair in FP32: D = 0, f = r.  From r² = 66 A on, A = a_i a_j,
// D is below e^-16.5 and 2 - D/2 is 2 to the last bit.  The derivative by A,
// which an atom needs whose radius is not clamped at 0.5 Å, is dropped from 160 A
// on (below e^-40 of the pair's energy).
constexpr float GB_FAR_FORCE = 66.0f, GB_FAR_BORN = 160.0f;

__device__ __forceinline__ double grad_screened_far(const DevParams &P, float r2, float qp) {
    const float rinv = rsqrtf(r2), r = r2 * rinv;
    const float kap = (float)P.kappa;
    const float edh = (float)P.coulomb_over_epsw * qp * rinv * __expf(-kap * r);
    const float f_dh = -edh * (rinv + kap) * rinv;
    const float egb = (float)P.gb_coef * qp * rinv;
    const float f_gb = -egb * __fdividef(1.0f, r2);
    return (double)f_dh + (double)f_gb;
}

// LJ + hard core inside sigma, FP64 with FP64 sigma / epsilon (the steep terms).
__device__ __forceinline__ double grad_contact(const DevParams &P, double r2d, double sig2, double sig64, double eps64) {
    const double s2 = sig2 / r2d, s6 = s2 * s2 * s2;
    double f = 4.0 * sqrt(eps64) * (6.0 * s6 - 12.0 * s6 * s6) / r2d;
    const double rc = sig64 * P.hard_frac, rc2 = rc * rc;
    if (r2d < rc2) {
        const double t2 = rc2 / r2d, t6 = t2 * t2 * t2, t12 = t6 * t6, x = t12 - 1.0;
        if (P.hard_scale * x * x < P.hard_cap) f += -24.0 * P.hard_scale * x * t12 / r2d;
    }
    return f;
}

// LJ outside sigma: s² in FP64, the powers in R.
template <typename R>
__device__ __forceinline__ double grad_lj(double r2d, double sig2, R eps_prod) {
    const R r2 = (R)r2d;
    if constexpr (sizeof(R) == 4) {
        const float rinv = rsqrtf(r2);
        const R s2 = (R)(sig2 * recip_from(r2d, rinv * rinv));
        const R s6 = s2 * s2 * s2;
        return (double)(4.0f * f_sqrt(eps_prod) * (6.0f * s6 - 12.0f * s6 * s6) * __fdividef(1.0f, r2));
    } else {
        const R s2 = (R)(sig2 / r2d);
        const R s6 = s2 * s2 * s2;
        return (double)((R)4 * m_sqrt(eps_prod) * ((R)6 * s6 - (R)12 * s6 * s6) / r2);
    }
}

// d/dr of hct(r; ri, rj) = 1/L - 1/U + P ln(L/U) / (4 ri² r²),
// L = max(|r - rj|, ri), U = r + rj, P = r² - rj² + ri² (:2007-2011).
template <typename R>
__device__ __forceinline__ R hct_deriv(R r, R r2, R ri, R rj) {
    const R U = r + rj;
    if (ri >= U) return (R)0;
    if constexpr (sizeof(R) == 4) {  // fast reciprocals, logf kept (see hct_term)
        const float d = fabsf(r - rj);
        float L, Lp;
        if (d > ri) {
            L = d;
            Lp = r > rj ? 1.0f : -1.0f;
        } else {
            L = ri;
            Lp = 0.0f;
        }
        const float rL = __fdividef(1.0f, L), rU = __fdividef(1.0f, U), rr = __fdividef(1.0f, r);
        const float Pp = r2 - rj * rj + ri * ri;
        const float Q = logf(L * rU);
        const float rden = __fdividef(0.25f, ri * ri * r2);
        const float T = Pp * Q * rden;
        const float dT = (2.0f * r * Q + Pp * (Lp * rL - rU)) * rden - 2.0f * T * rr;
        return -Lp * rL * rL + rU * rU + dT;
    }
    const R d = m_abs(r - rj);
    R L, Lp;
    if (d > ri) {
        L = d;
        Lp = r > rj ? (R)1 : (R)-1;
    } else {
        L = ri;
        Lp = (R)0;
    }
    const R Pp = r2 - rj * rj + ri * ri;
    const R Q = m_log(L / U);
    const R den = (R)4 * ri * ri * r2;
    const R T = Pp * Q / den;
    const R dT = ((R)2 * r * Q + Pp * (Lp / L - (R)1 / U)) / den - (R)2 * T / r;
    return -Lp / (L * L) + (R)1 / (U * U) + dT;
}

// 0.15^n.
__device__ __forceinline__ double pow015(int n) {
    double r = 1.0, b = 0.15;
    for (; n; n >>= 1) {
        if (n & 1) r *= b;
        b *= b;
    }
    return r;
}

// The SASA adjoint of a row with more entries within reach than the list of
// grad_pair_kernel holds (an unphysically dense row): the recurrence over the
// ordered half row twice, once to count the 0.85-branch entries, once for the
// adjoints.  One warp.
__device__ __noinline__ void grad_sasa_row(const DevParams &P, int i, int lane, const double *__restrict__ xyz,
                                           const double *__restrict__ prm64, int64_t beg, int64_t end,
                                           const uint32_t *__restrict__ half_cols, unsigned long long *__restrict__ fix,
                                           double &gx, double &gy, double &gz) {
    const double4 pi = ld_xyz(xyz, i);
    const double rsi = prm64[4 * (size_t)i + 1] + P.probe_r;
    const double cap_scale = 2.0 * 3.14159265358979323846 * rsi * rsi;
    const double base = P.gamma_sa * 3.14159265358979323846 * rsi;  // -dE/dcap * dcap/dr
    int n_frac = 0;
    for (int pass = 0; pass < 2; ++pass) {
        double sa = 4.0 * 3.14159265358979323846 * rsi * rsi;
        int seen = 0;
        for (int64_t k0 = beg; k0 < end; k0 += 32) {
            const int64_t k = k0 + lane;
            double cap = 0.0, dx = 0.0, dy = 0.0, dz = 0.0, r = 1.0;
            bool hit = false;
            int j = 0;
            if (k < end) {
                j = (int)(half_cols[k] & ALMA_IDX_MASK);
                const double4 pj = ld_xyz(xyz, j);
                dx = pi.x - pj.x;
                dy = pi.y - pj.y;
                dz = pi.z - pj.z;
                r = sqrt(dx * dx + dy * dy + dz * dz);
                const double dc = rsi + prm64[4 * (size_t)j + 1] + P.probe_r;
                if (r < dc) {
                    hit = true;
                    cap = cap_scale * ((dc - r) / (2.0 * rsi));
                }
            }
            // packed lane q holds the q-th hit; its adjoint goes back to the hit's own lane
            const unsigned m = __ballot_sync(0xffffffffu, hit);
            const int n = __popc(m);
            const double packed = sasa_pack(m, cap, lane);
            double pcoef = 0.0;
            for (int q = 0; q < n; ++q) {
                const double c = __shfl_sync(0xffffffffu, packed, q);
                if (c <= sa * 0.85) {
                    sa -= c;
                    if (pass == 1 && lane == q) pcoef = base * pow015(n_frac - seen);
                } else {
                    sa -= sa * 0.85;
                    ++seen;
                }
            }
            const double coef = __shfl_sync(0xffffffffu, pcoef, __popc(m & ((1u << lane) - 1u)));
            if (hit && coef != 0.0) {
                const double s = coef / r;
                gx += s * dx;
                gy += s * dy;
                gz += s * dz;
                fix_add(&fix[3 * (size_t)j], -s * dx);
                fix_add(&fix[3 * (size_t)j + 1], -s * dy);
                fix_add(&fix[3 * (size_t)j + 2], -s * dz);
            }
        }
        if (!(sa > 0.0)) return;  // max(0, sa) is flat here
        n_frac = seen;
    }
}

// Per-warp lists of the pair pass: the row's SASA entries (one row of a
// folded protein has 30-70), and near pairs (inside sigma, or reached by GB's
// exponential) waiting for 32.
constexpr int GRAD_SASA_LIST = 192;
struct GradBuf {
    double near_r2[64];  // squared distance
    int32_t near_j[64];
    int32_t sasa_j[GRAD_SASA_LIST];
    int32_t branch[GRAD_SASA_LIST];  // 0.85-branch entries before this one, -1: it took that branch itself
};

// A Born coefficient below this is taken as 0: its chain-rule terms (hct' is
// at most 1/L², a few hundred per row) stay under 1e-20 kcal/mol/Å, ten orders
// below the gradient's fixed-point parts.  Atoms that GB's exponential barely
// reaches have coefficients like e^-100.
constexpr double BORN_COEF_MIN = 1e-24;

// Warp per atom, 256 threads, 4 blocks per SM (2 in FP64).  The latency of the
// row's gathers bounds it, and the occupancy pays for a few spilled registers
// (65k atoms: 530 us with 3 blocks, 463 with 4, 471 with 5); an entry needs FP64 for its distance, and the
// FP64 square roots and divisions of the few SASA entries and contacts inside
// sigma run packed, 32 to a warp, instead of once per chunk with most lanes
// idle.  The SASA adjoint shares the row and its distances: as a kernel of
// its own over the half rows, with an FP64 square root and division for every
// entry, it took longer than the pair forces.  65k atoms, 39 M entries: 323 +
// 454 us in two kernels, 463 us in this one.
template <typename R, bool WIDE>
__global__ void __launch_bounds__(256, sizeof(R) == 4 ? 4 : 2) grad_pair_kernel(DevParams P, int natoms, const int32_t *__restrict__ atom_off, int nsys,
                                 const uint8_t *__restrict__ mask, const double *__restrict__ xyz,
                                 const float *__restrict__ prm, const double *__restrict__ prm64,
                                 const double *__restrict__ born, AlmaNL nl, int use_excl, double *__restrict__ grad,
                                 double *__restrict__ born_coef, unsigned long long *__restrict__ fix) {
    __shared__ GradBuf bufs[8];
    GradBuf &buf = bufs[threadIdx.x >> 5];
    const int i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (i >= natoms) return;
    if (mask && !mask[sys_of_atom(atom_off, nsys, i)]) return;
    R qi, ri, ei;
    load_prm<R>(prm, prm64, i, qi, ri, ei);
    const double4 pi = ld_pos<WIDE>(xyz, i);
    const double ri64 = prm64[4 * (size_t)i + 1], ei64 = prm64[4 * (size_t)i + 2];
    const double rsi = ri64 + P.probe_r;
    const float reach_i = (float)(rsi + P.probe_r);
    const double born_i = born[i];
    const R ai = (R)born_i;
    const float gb_far = born_i < 0.5 ? GB_FAR_BORN : GB_FAR_FORCE;
    double gx = 0.0, gy = 0.0, gz = 0.0, da = 0.0;
    int nsasa = 0, nnear = 0;
    const unsigned below = (1u << lane) - 1u;
    auto contacts = [&](int n) {
        if (lane >= n) return;
        const int j = buf.near_j[lane];
        const double4 pj = ld_pos<WIDE>(xyz, j);
        const double4 q = *reinterpret_cast<const double4 *>(prm64 + 4 * (size_t)j);
        const double r2 = buf.near_r2[lane], sig64 = ri64 + q.y, sig2 = sig64 * sig64;
        R qj, rj, ej;
        load_prm<R>(prm, prm64, j, qj, rj, ej);
        const double bj = born[j];
        double dEdA;
        double fr = grad_screened<R>(P, (R)r2, qi * qj, ai, (R)bj, dEdA);
        da += dEdA * bj;
        if (r2 < sig2) fr += grad_contact(P, r2, sig2, sig64, ei64 * q.z);
        else fr += grad_lj<R>(r2, sig2, ei * ej);
        gx += fr * (pi.x - pj.x);
        gy += fr * (pi.y - pj.y);
        gz += fr * (pi.z - pj.z);
    };
    const int64_t beg = nl.full_ptr[i], end = beg + nl.full_len[i];
    // the next entry is fetched while this one is evaluated, and an entry's
    // gathers are issued together (one dependent round trip per entry)
    uint32_t nxt = beg + lane < end ? nl.full_cols[beg + lane] : 0u;
    for (int64_t k0 = beg; k0 < end; k0 += 32) {
        const int64_t k = k0 + lane;
        bool hit = false, near = false;
        int j = 0;
        double r2 = 0.0;
        if (k < end) {
            const uint32_t ent = nxt;
            if (k + 32 < end) nxt = nl.full_cols[k + 32];
            j = (int)(ent & ALMA_IDX_MASK);
            const double4 pj = ld_pos<WIDE>(xyz, j);
            R qj, rj, ej;
            load_prm<R>(prm, prm64, j, qj, rj, ej);
            const double rj64 = prm64[4 * (size_t)j + 1];
            const double bj = born[j];
            const double dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
            r2 = dx * dx + dy * dy + dz * dz;
            const float r2f = (float)r2;
            hit = j > i && r2f < widened2(reach_i + (float)rj);
            if (!(use_excl && (ent & ALMA_EXCL_BIT)) && !(r2 > P.pair_cut2)) {
                if constexpr (sizeof(R) == 4) near = r2f < fmaxf(widened2(ri + rj), gb_far * (ai * (R)bj));
                else near = r2f < widened2((float)(ri + rj));
                if (!near) {
                    const double sig64 = ri64 + rj64;
                    double f;
                    if constexpr (sizeof(R) == 4) {
                        f = grad_screened_far(P, r2f, qi * qj);
                    } else {
                        double dEdA;
                        f = grad_screened<R>(P, (R)r2, qi * qj, ai, (R)bj, dEdA);
                        da += dEdA * bj;
                    }
                    const double fr = f + grad_lj<R>(r2, sig64 * sig64, ei * ej);
                    gx += fr * dx;
                    gy += fr * dy;
                    gz += fr * dz;
                }
            }
        }
        const unsigned mh = __ballot_sync(0xffffffffu, hit), mn = __ballot_sync(0xffffffffu, near);
        if (hit) {
            const int at = nsasa + __popc(mh & below);
            if (at < GRAD_SASA_LIST) buf.sasa_j[at] = j;
        }
        nsasa += __popc(mh);
        if (near) {
            const int at = nnear + __popc(mn & below);
            buf.near_r2[at] = r2;
            buf.near_j[at] = j;
        }
        nnear += __popc(mn);
        if (nnear >= 32) {
            __syncwarp();
            contacts(32);
            nnear -= 32;
            double a = 0.0;
            int jj = 0;
            if (lane < nnear) { a = buf.near_r2[32 + lane]; jj = buf.near_j[32 + lane]; }
            __syncwarp();
            if (lane < nnear) { buf.near_r2[lane] = a; buf.near_j[lane] = jj; }
            __syncwarp();
        }
    }
    __syncwarp();
    contacts(nnear);
    double sx = 0.0, sy = 0.0, sz = 0.0;  // SASA force on atom i
    if (nsasa > GRAD_SASA_LIST) {
        grad_sasa_row(P, i, lane, xyz, prm64, nl.half_ptr[i], nl.half_ptr[i] + nl.half_len[i], nl.half_cols, fix, sx,
                      sy, sz);
    } else if (nsasa > 0) {
        const double cap_scale = 2.0 * 3.14159265358979323846 * rsi * rsi;
        const double base = P.gamma_sa * 3.14159265358979323846 * rsi;  // -dE/dcap * dcap/dr
        double sa = 4.0 * 3.14159265358979323846 * rsi * rsi;
        int seen = 0;
        for (int b = 0; b < nsasa; b += 32) {
            double cap = -1.0;  // not within the FP64 reach: no entry
            if (b + lane < nsasa) {
                const int j = buf.sasa_j[b + lane];
                const double r = sqrt(d2_of(pi, ld_pos<WIDE>(xyz, j)));
                const double dc = rsi + prm64[4 * (size_t)j + 1] + P.probe_r;
                if (r < dc) cap = cap_scale * ((dc - r) / (2.0 * rsi));
            }
            const int n = min(32, nsasa - b);
            int mine = -1;
            for (int q = 0; q < n; ++q) {  // row order; the shuffles do not wait for sa
                const double c = __shfl_sync(0xffffffffu, cap, q);
                if (c < 0.0) continue;
                if (c <= sa * 0.85) {
                    sa -= c;
                    if (lane == q) mine = seen;
                } else {
                    sa -= sa * 0.85;
                    ++seen;
                }
            }
            if (b + lane < nsasa) buf.branch[b + lane] = mine;
        }
        if (sa > 0.0) {  // else max(0, sa) is flat
            for (int t = lane; t < nsasa; t += 32) {
                if (buf.branch[t] < 0) continue;
                const int j = buf.sasa_j[t];
                const double4 pj = ld_pos<WIDE>(xyz, j);
                const double dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
                const double s = base * pow015(seen - buf.branch[t]) / sqrt(dx * dx + dy * dy + dz * dz);
                sx += s * dx;
                sy += s * dy;
                sz += s * dz;
                fix_add(&fix[3 * (size_t)j], -s * dx);
                fix_add(&fix[3 * (size_t)j + 1], -s * dy);
                fix_add(&fix[3 * (size_t)j + 2], -s * dz);
            }
        }
    }
    gx = warp_sum(gx + sx);
    gy = warp_sum(gy + sy);
    gz = warp_sum(gz + sz);
    da = warp_sum(da);
    if (lane == 0) {
        *reinterpret_cast<double4 *>(grad + 4 * (size_t)i) = make_double4(gx, gy, gz, 0.0);
        const double c = born_i < 0.5 ? 0.5 * da * born_i * born_i : 0.0;
        born_coef[i] = fabs(c) >= BORN_COEF_MIN ? c : c != c ? c : 0.0;
    }
}

__device__ __forceinline__ double3 sub3(double4 a, double4 b) { return make_double3(a.x - b.x, a.y - b.y, a.z - b.z); }
__device__ __forceinline__ double3 cross3(double3 a, double3 b) {
    return make_double3(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
}
__device__ __forceinline__ double dot3(double3 a, double3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }

__device__ __forceinline__ void fix_add3(unsigned long long *fix, int i, double s, double3 v) {
    fix_add(&fix[3 * (size_t)i], s * v.x);
    fix_add(&fix[3 * (size_t)i + 1], s * v.y);
    fix_add(&fix[3 * (size_t)i + 2], s * v.z);
}

// Dihedral records and disulfide springs, one thread each.
__global__ void grad_bonded_kernel(DevParams P, const int32_t *__restrict__ atom_off, int nsys,
                                   const uint8_t *__restrict__ mask, const double *__restrict__ xyz, AlmaTopo t,
                                   int ndih, int nss, unsigned long long *__restrict__ fix) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r < ndih) {
        const int4 q = *reinterpret_cast<const int4 *>(t.dih_abcd + 4 * (size_t)r);
        if (mask && !mask[sys_of_atom(atom_off, nsys, q.x)]) return;
        const double4 A = ld_xyz(xyz, q.x), B = ld_xyz(xyz, q.y), Cc = ld_xyz(xyz, q.z), D = ld_xyz(xyz, q.w);
        const double3 b1 = sub3(A, B), b2 = sub3(Cc, B), b3 = sub3(D, Cc);
        const double3 n1 = cross3(b1, b2), n2 = cross3(b2, b3), m1 = cross3(n1, b2);
        const double x = dot3(n1, n2), y = dot3(m1, n2);
        const double phi = atan2(y, x);
        double dEdphi = 0.0;
        for (int k = t.term_off[r]; k < t.term_off[r + 1]; ++k) {
            const double n = (double)t.term_n[k];
            dEdphi -= t.term_v2[k] * n * sin(n * phi - t.term_gamma[k]);
        }
        // gradient of the true dihedral (Blondel & Karplus, J. Comput. Chem.
        // 17:1132, 1996) with F = a-b, G = b-c, H = d-c, then the map
        // phi_ref = atan2(L sin phi, cos phi), L = |b2|.
        const double3 F = b1, G = make_double3(-b2.x, -b2.y, -b2.z), H = b3;
        const double3 Av = cross3(F, G), Bv = cross3(H, G);
        const double A2 = dot3(Av, Av), B2 = dot3(Bv, Bv), Gn = sqrt(dot3(G, G));
        const double FG = dot3(F, G), HG = dot3(H, G);
        const double NN = dot3(n1, n1) * dot3(n2, n2);
        const double den = (x * x + y * y) / NN;  // cos^2 + L^2 sin^2
        const double sc = (y / Gn) * x / NN;       // sin cos
        const double sA = dEdphi * Gn / den, sB = dEdphi / den;
        // d(phi_ref) = (L d(phi) + sin cos dL) / den, d(phi) = -(BK terms)
        const double ka = Gn / A2, kb = Gn / B2, kfa = FG / (A2 * Gn), khb = HG / (B2 * Gn);
        fix_add3(fix, q.x, sA, make_double3(ka * Av.x, ka * Av.y, ka * Av.z));
        fix_add3(fix, q.w, -sA, make_double3(kb * Bv.x, kb * Bv.y, kb * Bv.z));
        const double3 gb = make_double3(ka * Av.x + kfa * Av.x - khb * Bv.x, ka * Av.y + kfa * Av.y - khb * Bv.y,
                                        ka * Av.z + kfa * Av.z - khb * Bv.z);
        const double3 gc = make_double3(-kfa * Av.x + khb * Bv.x - kb * Bv.x, -kfa * Av.y + khb * Bv.y - kb * Bv.y,
                                        -kfa * Av.z + khb * Bv.z - kb * Bv.z);
        const double3 u2 = make_double3(b2.x / Gn, b2.y / Gn, b2.z / Gn);  // dL/dc = b2/L = -dL/db
        fix_add3(fix, q.y, -sA, gb);
        fix_add3(fix, q.y, -sB * sc, u2);
        fix_add3(fix, q.z, -sA, gc);
        fix_add3(fix, q.z, sB * sc, u2);
        return;
    }
    const int k = r - ndih;
    if (k < nss) {
        const int i = t.ss_ij[2 * k], j = t.ss_ij[2 * k + 1];
        if (mask && !mask[sys_of_atom(atom_off, nsys, i)]) return;
        const double3 d = sub3(ld_xyz(xyz, i), ld_xyz(xyz, j));
        const double rr = sqrt(dot3(d, d));
        const double s = 2.0 * P.k_ss * (rr - P.r0_ss) / rr;
        fix_add3(fix, i, s, d);
        fix_add3(fix, j, -s, d);
    }
}

// Born-radius chain rule plus the final sum into grad.  The radii of about
// seven atoms in eight sit at the clamp, where the coefficient is 0: an entry's
// coefficient is read first, and the entries that count (all of an unclamped
// atom's row, an eighth of the others') are packed so that 32 of them share
// the two gathers and the HCT derivatives.  What is left is the latency of the
// coefficient gathers (6 blocks per SM 127 us, 4 blocks 157).  65k atoms, 39 M
// entries: 285 -> 127 us.
template <typename R, bool WIDE>
__global__ void __launch_bounds__(256, sizeof(R) == 4 ? 6 : 3) grad_born_kernel(int natoms, const int32_t *__restrict__ atom_off, int nsys,
                                 const uint8_t *__restrict__ mask, const double *__restrict__ xyz,
                                 const float *__restrict__ prm, const double *__restrict__ prm64,
                                 const int64_t *__restrict__ full_ptr, const int32_t *__restrict__ full_len,
                                 const uint32_t *__restrict__ full_cols, const double *__restrict__ born_coef,
                                 const unsigned long long *__restrict__ fix, double *__restrict__ grad) {
    __shared__ double buf_c[8][64];
    __shared__ int32_t buf_j[8][64];
    double *bc = buf_c[threadIdx.x >> 5];
    int32_t *bj = buf_j[threadIdx.x >> 5];
    const int i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (i >= natoms) return;
    if (mask && !mask[sys_of_atom(atom_off, nsys, i)]) return;
    auto radius = [&](int j) {
        if constexpr (sizeof(R) == 4) return prm[4 * (size_t)j + 1];
        else return prm64[4 * (size_t)j + 1];
    };
    const R ri = radius(i);
    const double4 pi = ld_pos<WIDE>(xyz, i);
    const double ci = born_coef[i];
    double gx = 0.0, gy = 0.0, gz = 0.0;
    auto evaluate = [&](int n) {
        if (lane >= n) return;
        const int j = bj[lane];
        const double cj = bc[lane];
        const R rj = radius(j);
        const double4 pj = ld_pos<WIDE>(xyz, j);
        const double dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
        const R r2 = (R)(dx * dx + dy * dy + dz * dz);
        const R r = f_sqrt(r2);
        double h = 0.0;
        if (ci != 0.0) h = ci * (double)hct_deriv<R>(r, r2, ri, rj);  // the same for the whole warp
        if (cj != 0.0) h += cj * (double)hct_deriv<R>(r, r2, rj, ri);
        double s;
        if constexpr (sizeof(R) == 4) s = h * recip_from((double)r, __fdividef(1.0f, r));
        else s = h / r;
        gx += s * dx;
        gy += s * dy;
        gz += s * dz;
    };
    int n = 0;
    const unsigned below = (1u << lane) - 1u;
    const int64_t beg = full_ptr[i], end = beg + full_len[i];
    // two chunks at a time: both entries, then both coefficients in flight
    for (int64_t k0 = beg; k0 < end; k0 += 64) {
        int j[2];
        double c[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int64_t k = k0 + 32 * u + lane;
            j[u] = k < end ? (int)(full_cols[k] & ALMA_IDX_MASK) : -1;
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) c[u] = j[u] >= 0 ? born_coef[j[u]] : 0.0;
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const bool counts = j[u] >= 0 && (ci != 0.0 || c[u] != 0.0);
            const unsigned m = __ballot_sync(0xffffffffu, counts);
            if (m == 0u) continue;
            if (counts) {
                const int at = n + __popc(m & below);
                bj[at] = j[u];
                bc[at] = c[u];
            }
            n += __popc(m);
            if (n >= 32) {
                __syncwarp();
                evaluate(32);
                n -= 32;
                int jj = 0;
                double cc = 0.0;
                if (lane < n) { jj = bj[32 + lane]; cc = bc[32 + lane]; }
                __syncwarp();
                if (lane < n) { bj[lane] = jj; bc[lane] = cc; }
                __syncwarp();
            }
        }
    }
    __syncwarp();
    evaluate(n);
    gx = warp_sum(gx);
    gy = warp_sum(gy);
    gz = warp_sum(gz);
    if (lane == 0) {
        double4 g = *reinterpret_cast<const double4 *>(grad + 4 * (size_t)i);
        g.x += gx + (double)(long long)fix[3 * (size_t)i] * FIX_INV;
        g.y += gy + (double)(long long)fix[3 * (size_t)i + 1] * FIX_INV;
        g.z += gz + (double)(long long)fix[3 * (size_t)i + 2] * FIX_INV;
        g.w = 0.0;
        *reinterpret_cast<double4 *>(grad + 4 * (size_t)i) = g;
    }
}

static size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

}  // namespace alma

using namespace alma;

extern "C" size_t alma_forces_workspace_bytes(int32_t natoms) {
    const size_t n = natoms > 0 ? (size_t)natoms : 1;
    return align256(sizeof(double) * n) + align256(sizeof(unsigned long long) * 3 * n);
}

extern "C" int alma_forces(const AlmaBatch *b, const AlmaTopo *t, const AlmaNL *nl, const AlmaParams *p,
                           int precision, const uint8_t *sys_mask, void *workspace, double *grad, void *stream) {
    if (!b || !nl || !p || !grad || !workspace || b->nsys <= 0 || b->natoms < 0)
        return alma_set_error(ALMA_EINVAL, "alma_forces: bad arguments");
    if (!b->atom_off || !b->xyz || !b->prm || !b->prm64 || !b->born || !nl->full_ptr || !nl->full_len ||
        !nl->full_cols || !nl->half_ptr || !nl->half_len || !nl->half_cols)
        return alma_set_error(ALMA_EINVAL, "alma_forces: null buffer");
    if (precision != ALMA_PREC_MIXED && precision != ALMA_PREC_FP64)
        return alma_set_error(ALMA_EINVAL, "alma_forces: precision must be ALMA_PREC_MIXED or ALMA_PREC_FP64");
    if (b->natoms == 0) return ALMA_OK;
    cudaStream_t st = (cudaStream_t)stream;
    const DevParams P = make_dev_params(*p);
    char *ws = (char *)workspace;
    double *born_coef = (double *)ws;
    unsigned long long *fix = (unsigned long long *)(ws + align256(sizeof(double) * (size_t)b->natoms));
    ALMA_CUDA_TRY(cudaMemsetAsync(fix, 0, sizeof(unsigned long long) * 3 * (size_t)b->natoms, st));
    const int wpb = 8;
    const int nb = (b->natoms + wpb - 1) / wpb;
    const int use_excl = t != nullptr;
    const bool wide = wide_ok(b->xyz), fp64 = precision == ALMA_PREC_FP64;
    auto pair = fp64 ? (wide ? grad_pair_kernel<double, true> : grad_pair_kernel<double, false>)
                     : (wide ? grad_pair_kernel<float, true> : grad_pair_kernel<float, false>);
    pair<<<nb, wpb * 32, 0, st>>>(P, b->natoms, b->atom_off, b->nsys, sys_mask, b->xyz, b->prm, b->prm64, b->born, *nl,
                                  use_excl, grad, born_coef, fix);
    int nlaunch = 2;
    if (t && (t->ndih > 0 || t->nss > 0)) {
        const int n = t->ndih + t->nss;
        grad_bonded_kernel<<<(n + 255) / 256, 256, 0, st>>>(P, b->atom_off, b->nsys, sys_mask, b->xyz, *t, t->ndih,
                                                            t->nss, fix);
        ++nlaunch;
    }
    auto bornk = fp64 ? (wide ? grad_born_kernel<double, true> : grad_born_kernel<double, false>)
                      : (wide ? grad_born_kernel<float, true> : grad_born_kernel<float, false>);
    bornk<<<nb, wpb * 32, 0, st>>>(b->natoms, b->atom_off, b->nsys, sys_mask, b->xyz, b->prm, b->prm64, nl->full_ptr,
                                   nl->full_len, nl->full_cols, born_coef, fix, grad);
    ALMA_LAUNCH_CHECK_N("alma_forces", nlaunch);
    return ALMA_OK;
}
