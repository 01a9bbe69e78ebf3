// Ensemble metrics over snapshots resident on the device: the mean Cα-Cα
// distance matrix and the contact-frequency matrix (compute_mean_dist_matrix
// and compute_contact_freq_matrix, analysis_ext.cpp:85-170; callers
// gui_main.py:1075-1200).  coords: [n_snaps, n_ca, 3] FP64.
//
// Tiles of 16 CELLS x 16 of the (i, j) matrix, CELLS per thread, upper triangle
// only (the lower one is its mirror).  A few snapshots of the tile's rows and
// columns sit in shared memory while the next are on their way, one barrier
// per stage.  Every cell sums its snapshots in order, as the reference's
// outer loop does, then scales by 1/n_snaps; that leaves the cells as the
// parallelism, and 512 per block keeps some twenty warps per SM busy at 600
// residues.  The mean is bound by the FP64 square roots, the contact frequency
// by shared-memory reads, of which four cells per thread need fewer each.  32 x 32
// tiles with a load and two barriers per snapshot took 1,227 us (mean) and 554 us
// (contacts) for 1,000 snapshots of 601 residues; now 450 and 298 us.
#include "alma_common.cuh"

namespace alma {

constexpr int AN_COLS = 16, AN_THREADS = AN_COLS * 16;

template <bool CONTACT, int CELLS>
__global__ void __launch_bounds__(AN_THREADS)
ensemble_matrix_kernel(const double *__restrict__ coords, int n_snaps, int n_ca, double cutoff2,
                       double *__restrict__ out) {
    constexpr int AN_ROWS = 16 * CELLS, AN_STAGE = 16 / CELLS;  // snapshots staged at a time
    constexpr int AN_SNAP = 3 * (AN_ROWS + AN_COLS);  // doubles of one staged snapshot
    constexpr int AN_LOADS = (AN_STAGE * AN_SNAP + AN_THREADS - 1) / AN_THREADS;
    __shared__ double buf[2][AN_STAGE][3][AN_ROWS + AN_COLS];  // rows, then columns, by component
    const int i0 = blockIdx.y * AN_ROWS, j0 = blockIdx.x * AN_COLS;
    if (j0 + AN_COLS <= i0) return;  // below the diagonal
    const int tx = threadIdx.x % AN_COLS, ty = threadIdx.x / AN_COLS;
    double acc[CELLS] = {}, next[AN_LOADS];
    // element q of a stage: snapshot, then the tile's coordinates as they lie
    // in memory (3 AN_ROWS of the rows, 3 AN_COLS of the columns)
    auto fetch = [&](int s0) {
#pragma unroll
        for (int u = 0; u < AN_LOADS; ++u) {
            const int q = u * AN_THREADS + (int)threadIdx.x, sn = s0 + q / AN_SNAP, e = q % AN_SNAP;
            const int at = e < 3 * AN_ROWS ? 3 * i0 + e : 3 * j0 + (e - 3 * AN_ROWS);
            next[u] = q < AN_STAGE * AN_SNAP && sn < n_snaps && at < 3 * n_ca ? coords[(size_t)sn * n_ca * 3 + at] : 0.0;
        }
    };
    auto store = [&](int b) {
#pragma unroll
        for (int u = 0; u < AN_LOADS; ++u) {
            const int q = u * AN_THREADS + (int)threadIdx.x, e = q % AN_SNAP;
            if (q < AN_STAGE * AN_SNAP) buf[b][q / AN_SNAP][e % 3][e / 3] = next[u];
        }
    };
    fetch(0);
    store(0);
    __syncthreads();
    int b = 0;
    for (int s0 = 0; s0 < n_snaps; s0 += AN_STAGE, b ^= 1) {
        const bool more = s0 + AN_STAGE < n_snaps;
        if (more) fetch(s0 + AN_STAGE);
        const int ns = min(AN_STAGE, n_snaps - s0);
        for (int k = 0; k < ns; ++k) {
            const double(*c)[AN_ROWS + AN_COLS] = buf[b][k];
            const double xj = c[0][AN_ROWS + tx], yj = c[1][AN_ROWS + tx], zj = c[2][AN_ROWS + tx];
#pragma unroll
            for (int r = 0; r < CELLS; ++r) {
                const int a = ty + 16 * r;
                const double dx = c[0][a] - xj, dy = c[1][a] - yj, dz = c[2][a] - zj;
                const double d2 = dx * dx + dy * dy + dz * dz;
                if (CONTACT) acc[r] += d2 < cutoff2 ? 1.0 : 0.0;
                else acc[r] += sqrt(d2);
            }
        }
        if (more) store(b ^ 1);  // its readers passed the barrier that ended the last round
        __syncthreads();
    }
    const double inv = n_snaps > 0 ? 1.0 / (double)n_snaps : 0.0;
#pragma unroll
    for (int r = 0; r < CELLS; ++r) {
        const int i = i0 + ty + 16 * r, j = j0 + tx;
        if (i >= n_ca || j >= n_ca) continue;
        if (j > i) {
            out[(size_t)i * n_ca + j] = acc[r] * inv;
            out[(size_t)j * n_ca + i] = acc[r] * inv;
        } else if (j == i) {
            out[(size_t)i * n_ca + i] = 0.0;
        }
    }
}

template <bool CONTACT>
static int ensemble_matrix(const double *coords, int32_t n_snaps, int32_t n_ca, double cutoff, double *out,
                           void *stream, const char *who) {
    if (n_snaps < 0 || n_ca < 0 || (n_ca > 0 && (!coords && n_snaps > 0)) || (n_ca > 0 && !out))
        return alma_set_error(ALMA_EINVAL, "%s: bad arguments", who);
    if (n_ca == 0) return ALMA_OK;
    const int nr = (n_ca + 31) / 32;
    if (nr > 65535) return alma_set_error(ALMA_EINVAL, "%s: n_ca too large", who);
    auto run = [&](auto kfn, int cells) {
        kfn<<<dim3((n_ca + AN_COLS - 1) / AN_COLS, (n_ca + 16 * cells - 1) / (16 * cells)), AN_THREADS, 0,
              (cudaStream_t)stream>>>(coords, n_snaps, n_ca, cutoff * cutoff, out);
    };
    // Contacts take four cells where that still leaves a block or so per SM (two
    // / four: 150 residues, 300 snapshots 42 / 60 us; 300 x 1,000 181 / 182;
    // 601 x 1,000 334 / 298; 1,500 x 1,000 1,248 / 1,084; 3,000 x 50 275 / 239);
    // the mean does not (601 x 1,000 450 / 776, 1,500 x 1,000 1,920 / 2,073).
    if constexpr (CONTACT) {
        if (n_ca >= 448) run(ensemble_matrix_kernel<true, 4>, 4);
        else run(ensemble_matrix_kernel<true, 2>, 2);
    } else {
        run(ensemble_matrix_kernel<false, 2>, 2);
    }
    ALMA_LAUNCH_CHECK(who);
    return ALMA_OK;
}

}  // namespace alma

using namespace alma;

extern "C" int alma_mean_dist_matrix(const double *coords, int32_t n_snaps, int32_t n_ca, double *out, void *stream) {
    return ensemble_matrix<false>(coords, n_snaps, n_ca, 0.0, out, stream, "alma_mean_dist_matrix");
}

extern "C" int alma_contact_freq_matrix(const double *coords, int32_t n_snaps, int32_t n_ca, double cutoff,
                                        double *out, void *stream) {
    return ensemble_matrix<true>(coords, n_snaps, n_ca, cutoff, out, stream, "alma_contact_freq_matrix");
}
