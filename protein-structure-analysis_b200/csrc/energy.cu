// Full-structure energy on the device: HCT Born radii, the ordered SASA
// term, the nonbonded pair sum, dihedral and disulfide terms, and a
// deterministic per-system reduction.
//
//   born   : warp per atom over its full row (every j with r² < 14²), FP64
//            accumulation of hct(i<-j) — the same set the reference's
//            symmetric half-list loop adds into sum[i] (physics_engine.cpp
//            :2024-2039), without float atomics.
//   pairs  : warp per atom over its half row, in one pass that also walks
//            the row in order for SASA (:2068-2083 — order dependent, so the
//            32 lanes compute the caps of 32 consecutive entries and the
//            recurrence sa -= min(0.85 sa, cap) is applied lane by lane),
//            and evaluates pair_e (:2148-2164) for non-excluded entries with
//            r² <= 12² (:2223-2232).
//   reduce : one cluster or CTA per system — pair and SASA sums in a fixed order,
//            plus the dihedral (:1912-1921) and disulfide (:1965-1974) terms.
#include <cooperative_groups.h>

#include "energy_core.cuh"

namespace alma {

namespace cg = cooperative_groups;

template <typename R, bool WIDE>
__global__ void born_kernel(int natoms, const int32_t *__restrict__ atom_off, int nsys, const uint8_t *__restrict__ mask,
                            const double *__restrict__ xyz, const float *__restrict__ prm,
                            const double *__restrict__ prm64, const int64_t *__restrict__ full_ptr,
                            const int32_t *__restrict__ full_len, const uint32_t *__restrict__ full_cols,
                            double *__restrict__ born) {
    const int i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (i >= natoms) return;
    if (mask && !mask[sys_of_atom(atom_off, nsys, i)]) return;
    born_atom<R, WIDE>(i, lane, xyz, prm, prm64, full_ptr, full_len, full_cols, born);
}

// Warp per atom: pair energy and SASA of row i.  atom_e[2*i] = pair sum of
// row i, atom_e[2*i+1] = gamma * max(0, sa_i).  Five 256-thread blocks per SM (48
// registers): the row gathers are latency bound and need the resident warps
// (65k atoms: 216 us with four blocks, 196 with five, 203 with six).
template <typename R, bool WIDE>
__global__ void __launch_bounds__(256, sizeof(R) == 4 ? 5 : 4) pair_sasa_kernel(DevParams P, int natoms, const int32_t *__restrict__ atom_off, int nsys,
                                 const uint8_t *__restrict__ mask, const double *__restrict__ xyz,
                                 const float *__restrict__ prm,
                                 const double *__restrict__ prm64, const double *__restrict__ born,
                                 const int64_t *__restrict__ half_ptr, const int32_t *__restrict__ half_len,
                                 const uint32_t *__restrict__ half_cols, int use_excl, double *__restrict__ atom_e,
                                 double *__restrict__ sasa_out) {
    __shared__ PairBuf buf[8];
    const int i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (i >= natoms) return;
    if (mask && !mask[sys_of_atom(atom_off, nsys, i)]) return;
    pair_sasa_atom<R, WIDE>(P, i, lane, xyz, prm, prm64, born, half_ptr, half_len, half_cols, use_excl,
                            buf[threadIdx.x >> 5], atom_e, sasa_out);
}

// The atoms' and records' terms of a system in eight strided shares, each
// summed by 256 threads, the shares' sums in order.  The dihedral records are
// the work (an FP64 atan2 and a cosine per term).  One system: a cluster of 8
// CTAs takes a share each and adds up through distributed shared memory (16k
// atoms: 52 -> 8.5 us, 65k: 234 -> 28).  Many small systems: a CTA each, which
// takes the shares one after the other.  The sums are the same either way, so
// a chain's terms do not depend on the batch.
constexpr int REDUCE_SHARES = 8;
constexpr int REDUCE_THREADS = 256;

template <int CTAS>
__global__ void __launch_bounds__(REDUCE_THREADS)
energy_reduce_kernel(DevParams P, const int32_t *__restrict__ atom_off, const double *__restrict__ xyz,
                     const double *__restrict__ atom_e, AlmaTopo t, int has_topo, const uint8_t *__restrict__ mask,
                     double *__restrict__ terms) {
    constexpr int PER = REDUCE_SHARES / CTAS, NW = REDUCE_THREADS / 32;  // shares per CTA
    __shared__ double sm[PER][4][NW], part[PER][4];
    const int rank = CTAS > 1 ? (int)cg::this_cluster().block_rank() : 0, s = blockIdx.x / CTAS;
    if (mask && !mask[s]) return;  // the whole cluster
    constexpr int stride = REDUCE_SHARES * REDUCE_THREADS;
    const int a0 = atom_off[s], a1 = atom_off[s + 1];
    const int d0 = has_topo ? t.dih_off[s] : 0, d1 = has_topo ? t.dih_off[s + 1] : 0;
    const int s0 = has_topo ? t.ss_off[s] : 0, s1 = has_topo ? t.ss_off[s + 1] : 0;
    // shares past the longest list are empty: their sums are 0
    const int longest = max(a1 - a0, max(d1 - d0, s1 - s0));
    const int used = PER > 1 ? min(PER, (longest + REDUCE_THREADS - 1) / REDUCE_THREADS) : 1;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int u = 0; u < used; ++u) {
        const int tid = (rank * PER + u) * REDUCE_THREADS + (int)threadIdx.x;
        double v[4] = {0.0, 0.0, 0.0, 0.0};  // pairs, SASA, dihedrals, disulfides
        for (int i = a0 + tid; i < a1; i += stride) {
            v[0] += atom_e[2 * (size_t)i];
            v[1] += atom_e[2 * (size_t)i + 1];
        }
        for (int r = d0 + tid; r < d1; r += stride) v[2] += dih_record_energy(xyz, t, r);
        for (int k = s0 + tid; k < s1; k += stride) {
            const double dr = sqrt(dist2(xyz, t.ss_ij[2 * k], t.ss_ij[2 * k + 1])) - P.r0_ss;
            v[3] += P.k_ss * dr * dr;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            v[k] = warp_sum(v[k]);
            if (lane == 0) sm[u][k][wid] = v[k];
        }
    }
    __syncthreads();
    if (threadIdx.x < 4 * used) {
        const int u = (int)threadIdx.x >> 2, k = threadIdx.x & 3;
        double q = 0.0;
        for (int w = 0; w < NW; ++w) q += sm[u][k][w];
        part[u][k] = q;
    }
    if constexpr (CTAS > 1) cg::this_cluster().sync();
    else __syncthreads();
    if (rank == 0 && threadIdx.x == 0) {
        double e[4] = {0.0, 0.0, 0.0, 0.0};
        for (int k = 0; k < 4; ++k) {
            if constexpr (CTAS > 1)
                for (int r = 0; r < CTAS; ++r) e[k] += cg::this_cluster().map_shared_rank(&part[0][0], r)[k];
            else
                for (int u = 0; u < used; ++u) e[k] += part[u][k];
        }
        const double sasa = (a1 > a0) ? P.beta_sa + e[1] : 0.0;
        double *o = terms + 5 * (size_t)s;
        o[0] = sasa;
        o[1] = e[2];
        o[2] = e[3];
        o[3] = e[0];
        o[4] = sasa + e[2] + e[3] + e[0];
    }
    if constexpr (CTAS > 1) cg::this_cluster().sync();  // no CTA leaves before its partials are read
}

}  // namespace alma

using namespace alma;

static int check_batch(const AlmaBatch *b, const char *who) {
    if (!b || b->nsys <= 0 || b->natoms < 0 || !b->atom_off || !b->xyz || !b->prm || !b->prm64 || !b->born)
        return alma_set_error(ALMA_EINVAL, "%s: bad batch", who);
    return ALMA_OK;
}

extern "C" int alma_born_radii(const AlmaBatch *b, const AlmaNL *nl, const AlmaParams *p, int prec,
                               const uint8_t *sys_mask, void *stream) {
    int rc = check_batch(b, "alma_born_radii");
    if (rc) return rc;
    if (!nl || !nl->full_ptr || !nl->full_cols || !p) return alma_set_error(ALMA_EINVAL, "alma_born_radii: null");
    if (b->natoms == 0) return ALMA_OK;
    cudaStream_t st = (cudaStream_t)stream;
    const int wpb = 8, nb = (b->natoms + wpb - 1) / wpb;
    const bool wide = wide_ok(b->xyz);
    auto kfn = prec == ALMA_PREC_FP64 ? (wide ? born_kernel<double, true> : born_kernel<double, false>)
                                      : (wide ? born_kernel<float, true> : born_kernel<float, false>);
    kfn<<<nb, wpb * 32, 0, st>>>(b->natoms, b->atom_off, b->nsys, sys_mask, b->xyz, b->prm, b->prm64, nl->full_ptr,
                                 nl->full_len, nl->full_cols, b->born);
    ALMA_LAUNCH_CHECK("alma_born_radii");
    return ALMA_OK;
}

extern "C" int alma_energy(const AlmaBatch *b, const AlmaTopo *t, const AlmaNL *nl, const AlmaParams *p, int prec,
                           const uint8_t *sys_mask, double *atom_e, double *terms, void *stream) {
    int rc = check_batch(b, "alma_energy");
    if (rc) return rc;
    if (!nl || !nl->half_ptr || !nl->half_cols || !p || !atom_e || !terms)
        return alma_set_error(ALMA_EINVAL, "alma_energy: null argument");
    cudaStream_t st = (cudaStream_t)stream;
    const DevParams P = make_dev_params(*p);
    if (b->natoms > 0) {
        const int wpb = 8, nb = (b->natoms + wpb - 1) / wpb;
        const int use_excl = t != nullptr;
        const bool wide = wide_ok(b->xyz);
        auto kfn = prec == ALMA_PREC_FP64 ? (wide ? pair_sasa_kernel<double, true> : pair_sasa_kernel<double, false>)
                                          : (wide ? pair_sasa_kernel<float, true> : pair_sasa_kernel<float, false>);
        kfn<<<nb, wpb * 32, 0, st>>>(P, b->natoms, b->atom_off, b->nsys, sys_mask, b->xyz, b->prm, b->prm64, b->born,
                                     nl->half_ptr, nl->half_len, nl->half_cols, use_excl, atom_e, b->sasa);
    }
    AlmaTopo tt;
    if (t) tt = *t;
    else memset(&tt, 0, sizeof(tt));
    // A CTA per system where its serial shares are shorter than the queue of
    // clusters: mean atoms up to 16 per system of the batch (64 x 1,089 atoms: 9.0 us
    // either way; 300 x 2.4k: 20.7 against 29.9, 400 x 1,089: 12 and 36, 2,000 x
    // 324: 21 and 137; 100 x 2.4k: 19.2 against 12.5, 128 x 4.9k: 26 and 18).
    const bool one = (int64_t)b->natoms <= 16 * (int64_t)b->nsys * b->nsys;
    if (one)
        energy_reduce_kernel<1><<<b->nsys, REDUCE_THREADS, 0, st>>>(P, b->atom_off, b->xyz, atom_e, tt, t != nullptr,
                                                                    sys_mask, terms);
    else
        ALMA_CUDA_TRY(alma_launch_cluster(energy_reduce_kernel<REDUCE_SHARES>, (unsigned)b->nsys * REDUCE_SHARES,
                                          REDUCE_THREADS, REDUCE_SHARES, (size_t)0, st, P, b->atom_off, b->xyz, atom_e,
                                          tt, t != nullptr, sys_mask, terms));
    ALMA_LAUNCH_CHECK_N("alma_energy", b->natoms > 0 ? 2 : 1);
    return ALMA_OK;
}
