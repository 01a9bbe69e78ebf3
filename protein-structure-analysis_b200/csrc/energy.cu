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
//   reduce : one cluster per system — pair and SASA sums in a fixed order,
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

// One cluster of 8 CTAs per system: the atoms' and records' terms strided over
// the cluster, CTA partials summed in rank order through distributed shared
// memory.  The dihedral records are the work (an FP64 atan2 and a cosine per
// term): one CTA took 52 us at 16k atoms and 234 us at 65k, the cluster
// 8.5 and 28 us.  Always 8 CTAs, so that a chain's sums are the same
// alone and in a batch.
constexpr int REDUCE_CTAS = 8;
constexpr int REDUCE_THREADS = 256;

__global__ void __launch_bounds__(REDUCE_THREADS)
energy_reduce_kernel(DevParams P, const int32_t *__restrict__ atom_off, const double *__restrict__ xyz,
                     const double *__restrict__ atom_e, AlmaTopo t, int has_topo, const uint8_t *__restrict__ mask,
                     double *__restrict__ terms) {
    __shared__ double sm[4][REDUCE_THREADS / 32], part[4];
    cg::cluster_group cl = cg::this_cluster();
    const int rank = (int)cl.block_rank(), s = blockIdx.x / REDUCE_CTAS;
    if (mask && !mask[s]) return;  // the whole cluster
    const int tid = rank * REDUCE_THREADS + (int)threadIdx.x, nthr = REDUCE_CTAS * REDUCE_THREADS;
    const int a0 = atom_off[s], a1 = atom_off[s + 1];
    double v[4] = {0.0, 0.0, 0.0, 0.0};  // pairs, SASA, dihedrals, disulfides
    for (int i = a0 + tid; i < a1; i += nthr) {
        v[0] += atom_e[2 * (size_t)i];
        v[1] += atom_e[2 * (size_t)i + 1];
    }
    if (has_topo) {
        for (int r = t.dih_off[s] + tid; r < t.dih_off[s + 1]; r += nthr) v[2] += dih_record_energy(xyz, t, r);
        for (int k = t.ss_off[s] + tid; k < t.ss_off[s + 1]; k += nthr) {
            const double dr = sqrt(dist2(xyz, t.ss_ij[2 * k], t.ss_ij[2 * k + 1])) - P.r0_ss;
            v[3] += P.k_ss * dr * dr;
        }
    }
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        v[k] = warp_sum(v[k]);
        if (lane == 0) sm[k][wid] = v[k];
    }
    __syncthreads();
    if (threadIdx.x < 4) {
        double q = 0.0;
        for (int w = 0; w < REDUCE_THREADS / 32; ++w) q += sm[threadIdx.x][w];
        part[threadIdx.x] = q;
    }
    cl.sync();
    if (rank == 0 && threadIdx.x == 0) {
        double e[4];
        for (int k = 0; k < 4; ++k) {
            e[k] = 0.0;
            for (int r = 0; r < REDUCE_CTAS; ++r) e[k] += cl.map_shared_rank(part, r)[k];
        }
        const double sasa = (a1 > a0) ? P.beta_sa + e[1] : 0.0;
        double *o = terms + 5 * (size_t)s;
        o[0] = sasa;
        o[1] = e[2];
        o[2] = e[3];
        o[3] = e[0];
        o[4] = sasa + e[2] + e[3] + e[0];
    }
    cl.sync();  // no CTA leaves before its partials are read
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
    ALMA_CUDA_TRY(alma_launch_cluster(energy_reduce_kernel, (unsigned)b->nsys * REDUCE_CTAS, REDUCE_THREADS,
                                      REDUCE_CTAS, (size_t)0, st, P, b->atom_off, b->xyz, atom_e, tt, t != nullptr,
                                      sys_mask, terms));
    ALMA_LAUNCH_CHECK_N("alma_energy", b->natoms > 0 ? 2 : 1);
    return ALMA_OK;
}
