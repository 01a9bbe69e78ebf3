// Neighbor-list build on the device.
//
// Reproduces NeighborList::build (physics_engine.cpp:293-342) bit-exactly,
// including row order: a 14 Å+1e-6 cubic cell grid over the system's
// bounding box padded by one cell, atoms binned by floor((x-lo)/cs), and
// each row listing the atoms of the 27 neighbour cells in (dz, dy, dx)
// order, ascending atom index inside a cell, keeping r² < 14² (FP64).
// The half row keeps j > i (the reference's nb[i]); the full row keeps every
// j != i (used by Born radii and the move kernels, where the order is
// irrelevant).  Each entry carries the 1-2/1-3/SS exclusion flag in bit 31.
//
// Three launches, all stream-ordered, no host sync:
//   cells : one cluster per system — FP64 bounding box, grid shape, cell
//           counts, cell starts, atoms scattered into their cells
//   order : thread per atom — its rank in its cell (ascending index), and the
//           cell-ordered copy of positions that the row scan streams
//   rows  : warp per one or two neighbouring atoms — one scan of the 27 cells
//           marks the candidates, then each row is staged in shared memory,
//           takes space in the system's regions and is written
// Every stage honours an optional per-system mask, so systems can be
// rebuilt independently (the MC driver rebuilds only chains that drifted).
#include <cooperative_groups.h>

#include "alma_common.cuh"
#include "nl_core.cuh"

namespace alma {

namespace cg = cooperative_groups;

struct NLWork {
    SysGrid *grid;        // [nsys]; ncell = 0: the grid did not fit
    int32_t *cell_of;     // [natoms] local cell index
    int32_t *cell_end;    // [max_cells] counts, then fill positions, then ends
    int32_t *scattered;   // [natoms] atoms by cell, any order within a cell
    int32_t *cell_atoms;  // [natoms] atoms by cell, ascending within a cell
    float4 *cell_pos;     // [natoms + 32] per slot: FP32 position from the box centre, its square
    float4 *cell_atom;    // [natoms] per slot: the same position, R*
    unsigned long long *total_cells;  // [1] cells handed out
};

static size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

static size_t carve(NLWork *w, char *base, int32_t nsys, int32_t natoms, int64_t max_cells) {
    size_t off = 0;
    auto take = [&](size_t bytes) {
        char *p = base ? base + off : nullptr;
        off += align256(bytes);
        return p;
    };
    NLWork t;
    t.grid = (SysGrid *)take(sizeof(SysGrid) * (size_t)(nsys > 0 ? nsys : 1));
    t.cell_of = (int32_t *)take(sizeof(int32_t) * (size_t)natoms);
    t.cell_end = (int32_t *)take(sizeof(int32_t) * (size_t)max_cells);
    t.scattered = (int32_t *)take(sizeof(int32_t) * (size_t)natoms);
    t.cell_atoms = (int32_t *)take(sizeof(int32_t) * (size_t)natoms);
    t.cell_pos = (float4 *)take(sizeof(float4) * ((size_t)natoms + 32));  // the scan reads whole chunks of 32
    t.cell_atom = (float4 *)take(sizeof(float4) * (size_t)natoms);
    t.total_cells = (unsigned long long *)take(sizeof(unsigned long long));
    if (w) *w = t;
    return off;
}

// Box centre of a grid: the origin of the FP32 copy of its atoms.
__device__ __forceinline__ double3 grid_centre(const SysGrid &g) {
    return make_double3(g.xlo + 0.5 * g.nx * g.cs, g.ylo + 0.5 * g.ny * g.cs, g.zlo + 0.5 * g.nz * g.cs);
}

// One cluster of CL CTAs per system: box and grid (physics_engine.cpp
// :299-316), then count, scan and scatter of its atoms.  The per-system work
// is a few dependent passes over its atoms and cells, so it runs as one
// launch with cluster barriers instead of eight launches and two memsets over
// all cells (one 65k-atom system: 125 us in eight kernels, of which the
// bounding box by one CTA took 91; 33 us here).  Minima, maxima, counts
// and cell contents do not depend on CL.
constexpr int CELLS_THREADS = 512;

template <int CL>
__global__ void __launch_bounds__(CELLS_THREADS)
nl_cells_kernel(const int32_t *__restrict__ atom_off, const uint8_t *__restrict__ mask,
                const double *__restrict__ xyz, double nl_rcut2, int64_t max_cells, SysGrid *__restrict__ grid,
                unsigned long long *total_cells, int32_t *cell_of, int32_t *cell_end, int32_t *__restrict__ scattered,
                int64_t *__restrict__ need, uint32_t *status) {
    constexpr int NW = CELLS_THREADS / 32, ITEMS = 4;
    __shared__ double red[6][NW], box[6];
    __shared__ long long cells_at;  // rank 0: first cell of the system, -1 when the grid does not fit
    __shared__ int slice_total, warp_tot[NW];
    const int rank = CL > 1 ? (int)cg::this_cluster().block_rank() : 0;
    const int s = blockIdx.x / CL;
    if (mask && !mask[s]) return;  // the whole cluster
    auto sync = [] {
        if constexpr (CL > 1) cg::this_cluster().sync();
        else __syncthreads();
    };
    auto peer = [](auto *p, int r) {
        if constexpr (CL > 1) return cg::this_cluster().map_shared_rank(p, r);
        else return p;
    };
    const int a0 = atom_off[s], a1 = atom_off[s + 1];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int tid = rank * CELLS_THREADS + (int)threadIdx.x, nthr = CL * CELLS_THREADS;
    // bounding box
    double mn[3] = {1e300, 1e300, 1e300}, mx[3] = {-1e300, -1e300, -1e300};
    for (int i = a0 + tid; i < a1; i += nthr) {
        const double4 p = ld_xyz(xyz, i);
        mn[0] = fmin(mn[0], p.x); mx[0] = fmax(mx[0], p.x);
        mn[1] = fmin(mn[1], p.y); mx[1] = fmax(mx[1], p.y);
        mn[2] = fmin(mn[2], p.z); mx[2] = fmax(mx[2], p.z);
    }
    for (int d = 0; d < 3; ++d) {
        for (int o = 16; o > 0; o >>= 1) {
            mn[d] = fmin(mn[d], __shfl_xor_sync(0xffffffffu, mn[d], o));
            mx[d] = fmax(mx[d], __shfl_xor_sync(0xffffffffu, mx[d], o));
        }
        if (lane == 0) { red[d][wid] = mn[d]; red[3 + d][wid] = mx[d]; }
    }
    __syncthreads();
    if (threadIdx.x < 6) {
        double v = red[threadIdx.x][0];
        for (int w = 1; w < NW; ++w)
            v = threadIdx.x < 3 ? fmin(v, red[threadIdx.x][w]) : fmax(v, red[threadIdx.x][w]);
        box[threadIdx.x] = v;
    }
    sync();
    double lo[3], hi[3];
    for (int d = 0; d < 3; ++d) {
        lo[d] = *peer(&box[d], 0);
        hi[d] = *peer(&box[3 + d], 0);
        for (int r = 1; r < CL; ++r) {
            lo[d] = fmin(lo[d], *peer(&box[d], r));
            hi[d] = fmax(hi[d], *peer(&box[3 + d], r));
        }
    }
    SysGrid g = grid_from_box(lo, hi, nl_rcut2, a1 - a0);
    if (rank == 0 && threadIdx.x == 0) {
        // (the product in FP64 first: a box that far out of range does not fit in any case)
        long long at = -1;
        if ((double)g.nx * g.ny * g.nz <= (double)max_cells) {
            at = (long long)atomicAdd(total_cells, (unsigned long long)g.ncell);
            if (at + g.ncell > max_cells) at = -1;
        }
        if (at < 0) set_status(status, ALMA_ST_CELL_OVERFLOW);
        cells_at = at;
        g.cell_off = at < 0 ? 0 : at;
        g.ncell = at < 0 ? 0 : g.ncell;
        grid[s] = g;
        for (int k = 0; k < 4; ++k) need[4 * (size_t)s + k] = 0;  // the row kernel counts here
    }
    sync();
    const long long at = *peer(&cells_at, 0);
    if (at < 0) {
        sync();  // rank 0 stays until every CTA has read its word
        return;
    }
    const int ncell = (int)g.ncell;  // <= max_cells, and a cell index is 32-bit
    int32_t *end = cell_end + at;
    for (int c = tid; c < ncell; c += nthr) end[c] = 0;
    sync();
    for (int i = a0 + tid; i < a1; i += nthr) {
        const int c = cell_of_point(g, ld_xyz(xyz, i));
        cell_of[i] = c;
        atomicAdd(&end[c], 1);
    }
    sync();
    // counts -> first slots: each CTA scans a slice of the cells behind the
    // totals of the slices before it
    const int per = (ncell + CL - 1) / CL, c0 = min(ncell, rank * per), c1 = min(ncell, c0 + per);
    if constexpr (CL > 1) {
        int sum = 0;
        for (int c = c0 + (int)threadIdx.x; c < c1; c += CELLS_THREADS) sum += end[c];
        sum = __reduce_add_sync(0xffffffffu, sum);
        if (lane == 0) warp_tot[wid] = sum;
        __syncthreads();
        if (threadIdx.x == 0) {
            int t = 0;
            for (int w = 0; w < NW; ++w) t += warp_tot[w];
            slice_total = t;
        }
        sync();
    }
    int carry = a0;
    for (int r = 0; r < rank; ++r) carry += *peer(&slice_total, r);
    for (int b0 = c0; b0 < c1; b0 += CELLS_THREADS * ITEMS) {
        int v[ITEMS], sum = 0;
#pragma unroll
        for (int k = 0; k < ITEMS; ++k) {
            const int c = b0 + (int)threadIdx.x * ITEMS + k;
            v[k] = c < c1 ? end[c] : 0;
            sum += v[k];
        }
        int inc = sum;
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += u;
        }
        __syncthreads();  // the warp totals of the last chunk have been read
        if (lane == 31) warp_tot[wid] = inc;
        __syncthreads();
        int at_ = carry + inc - sum;
        for (int w = 0; w < NW; ++w) {
            const int t = warp_tot[w];
            if (w < wid) at_ += t;
            carry += t;
        }
#pragma unroll
        for (int k = 0; k < ITEMS; ++k) {
            const int c = b0 + (int)threadIdx.x * ITEMS + k;
            if (c < c1) end[c] = at_;
            at_ += v[k];
        }
    }
    sync();
    for (int i = a0 + tid; i < a1; i += nthr) scattered[atomicAdd(&end[cell_of[i]], 1)] = i;
    // (every slot advanced by its cell's count: end[] now holds the cell ends)
}

// Thread per atom: its place in its cell is the number of smaller indices
// there (the reference pushes atoms in index order).  The threads of a warp
// mostly share a cell, so the reads are broadcasts.
__global__ void __launch_bounds__(256)
nl_order_kernel(const int32_t *__restrict__ atom_off, int nsys, int natoms, const uint8_t *__restrict__ mask,
                const SysGrid *__restrict__ grid, const int32_t *__restrict__ cell_of,
                const int32_t *__restrict__ cell_end, const int32_t *__restrict__ scattered,
                const double *__restrict__ xyz, const double *__restrict__ prm64, int32_t *__restrict__ cell_atoms,
                float4 *__restrict__ cell_pos, float4 *__restrict__ cell_atom) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= natoms) return;
    const int s = sys_of_atom(atom_off, nsys, i);
    if (mask && !mask[s]) return;
    const SysGrid g = grid[s];
    if (g.ncell == 0) return;
    const CellEnds cells{cell_end + g.cell_off, atom_off[s]};
    int64_t beg, end;
    cells(cell_of[i], beg, end);
    int at = (int)beg;
#pragma unroll 8
    for (int q = (int)beg; q < (int)end; ++q) at += scattered[q] < i;
    const double4 p = ld_xyz(xyz, i);
    const double3 o = grid_centre(g);
    const float x = (float)(p.x - o.x), y = (float)(p.y - o.y), z = (float)(p.z - o.z);
    cell_atoms[at] = i;
    cell_pos[at] = make_float4(x, y, z, x * x + y * y + z * z);
    cell_atom[at] = make_float4(x, y, z, prm64 ? (float)prm64[4 * (size_t)i + 1] : 0.0f);
}

// Row scan.  The candidates of an atom are the atoms of 27 cells: nine runs
// of three x-neighbours, each contiguous in the cell-ordered copy and already
// in the reference's scan order.  A warp takes G consecutive slots (atoms of
// one cell, or of neighbouring cells of one run: the run is then wider, which
// only adds candidates) and streams the runs once for all of them:
//   scan   |q|² - 2 p.q < 14² - |p|² in three FP32 FMAs per candidate, with a
//          margin that covers their rounding; the ballot of a chunk goes to
//          shared memory, chunks without a candidate are dropped
//   stage  the bits of each atom's masks become a list of slots
//   decide per staged slot, all lanes busy: the FP32 distance (coordinates
//          relative to the box centre), FP64 within fp32_margin2 of a cutoff,
//          the exclusion bit, the SASA reach — the rows are those of the FP64
//          tests bit for bit
//   write  space from the system's counters (one atomic per row kind, which
//          are also the entry counts), then the four rows, ballot-compacted
// Issue bounds it; shared memory lets eight blocks, 32 warps, on an SM.  The scan
// before this one compacted every chunk of 27 separate cells as it went, about
// 12,000 issue slots per atom at 600 neighbours.  65k atoms: 1,010 -> 431 us; 48 x
// 4.8k atoms: 1,892 -> 934 us.  Rows sit in their system's region in any order; a
// row that would overflow it is not written and raises the flag.
constexpr int NL_STAGE = 1280;  // staged entries of a row; a longer one is staged in parts
constexpr int NL_CHUNKS = 160;  // chunks of 32 candidates that hold one within reach; more are scanned in FP64
constexpr int NL_WARPS = 4;
constexpr uint32_t NL_SHORT_BIT = 0x40000000u;  // staging only: the pair is within SASA reach
constexpr uint32_t NL_DROPPED = 0xffffffffu;    // staging only: not an entry (2^30 - 2 is the largest index)

template <int G>
struct RowSmem {
    uint32_t stage[NL_STAGE];
    uint32_t bits[G][NL_CHUNKS];
    int32_t base[NL_CHUNKS];
};

// Space for the rows of atom i (n: entries per row kind in lanes 0-3): the
// offset of kind k in lane k, or false when a region is full.
__device__ __forceinline__ bool take_rows(const AlmaNL &nl, int s, int n, int lane, int nkind, int64_t &off,
                                          uint32_t *status) {
    bool fits = true;
    if (lane < nkind) {
        const int64_t *b = lane == 0 ? nl.full_base : lane == 1 ? nl.half_base : lane == 2 ? nl.sfull_base
                                                                                           : nl.shalf_base;
        const int64_t o = (int64_t)atomicAdd(reinterpret_cast<unsigned long long *>(nl.need + 4 * (size_t)s + lane),
                                             (unsigned long long)n);
        const int64_t beg = b[s];
        off = beg + o;
        fits = off + n <= b[s + 1];
    }
    if (__all_sync(0xffffffffu, fits)) return true;
    if (lane == 0) set_status(status, ALMA_ST_NL_OVERFLOW);
    return false;
}

__device__ __forceinline__ void set_rows(const AlmaNL &nl, int i, int n, int lane, int nkind, int64_t off) {
    if (lane < nkind) {
        (lane == 0 ? nl.full_ptr : lane == 1 ? nl.half_ptr : lane == 2 ? nl.sfull_ptr : nl.shalf_ptr)[i] = off;
        (lane == 0 ? nl.full_len : lane == 1 ? nl.half_len : lane == 2 ? nl.sfull_len : nl.shalf_len)[i] = n;
    }
}

template <int G>
__global__ void __launch_bounds__(NL_WARPS * 32, 8)
nl_rows_kernel(const int32_t *__restrict__ atom_off, int nsys, int natoms, const uint8_t *__restrict__ mask,
               const double *__restrict__ xyz, double rcut2, const SysGrid *__restrict__ grid,
               const int32_t *__restrict__ cell_of, const int32_t *__restrict__ cell_end,
               const int32_t *__restrict__ cell_atoms, const float4 *__restrict__ cell_pos,
               const float4 *__restrict__ cell_atom, const double *__restrict__ prm64, double reach_pad,
               const int64_t *__restrict__ excl_ptr, const int32_t *__restrict__ excl_cols,
               const uint32_t *__restrict__ excl_win, AlmaNL nl, uint32_t *status) {
    __shared__ RowSmem<G> smem[NL_WARPS];
    RowSmem<G> &W = smem[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const int p0 = (blockIdx.x * NL_WARPS + (threadIdx.x >> 5)) * G;
    if (p0 >= natoms) return;
    const bool shorts = nl.sfull_cols != nullptr;
    const int nkind = shorts ? 4 : 2;
    // lane g < G: the atom of slot p0 + g and its cell
    int my_s = -1, my_i = 0, my_cx = 0, my_row = -1;
    if (lane < G && p0 + lane < natoms) {
        const int s = sys_of_atom(atom_off, nsys, p0 + lane);
        if ((!mask || mask[s]) && grid[s].ncell > 0) {
            my_s = s;
            my_i = cell_atoms[p0 + lane];
            const int c = cell_of[my_i], nx = grid[s].nx;
            my_cx = c % nx;
            my_row = c / nx;
        }
    }
    unsigned todo = __ballot_sync(0xffffffffu, my_s >= 0);
    while (todo) {
        const int lead = __ffs(todo) - 1;
        const int s = __shfl_sync(0xffffffffu, my_s, lead), row = __shfl_sync(0xffffffffu, my_row, lead);
        const bool mine = my_s == s && my_row == row;
        const unsigned mem = __ballot_sync(0xffffffffu, mine) & todo;
        todo &= ~mem;
        const SysGrid g = grid[s];
        const CellEnds cells{cell_end + g.cell_off, atom_off[s]};
        const int x0 = max(0, __reduce_min_sync(0xffffffffu, mine ? my_cx : 0x7fffffff) - 1);
        const int x1 = min(g.nx - 1, __reduce_max_sync(0xffffffffu, mine ? my_cx : -1) + 1);
        // lane r < 9: run r in (dz, dy) order
        int rbeg = 0, rend = 0;
        if (lane < 9) {
            const int y = row % g.ny + lane % 3 - 1, z = row / g.ny + lane / 3 - 1;
            if (y >= 0 && y < g.ny && z >= 0 && z < g.nz) {
                const int64_t c = (int64_t)g.nx * (y + (int64_t)g.ny * z);
                rbeg = cells.beg(c + x0);
                rend = cells.end_[c + x1];
            }
        }
        // |p|² and the products round to within 2^-24 of terms up to 3/4
        // E² (E the longest side): 16 roundings of that size, twice over
        const float ext = (float)(fmax(g.nx, fmax(g.ny, g.nz)) * g.cs);
        const float m2 = g.margin2, cut_lo = (float)rcut2 - m2, cut_hi = (float)rcut2 + m2;
        const float cut_scan = cut_hi + 32.0f * 0.75f * 5.9604645e-8f * ext * ext;
        float ax[G], ay[G], az[G], thr[G];
#pragma unroll
        for (int a = 0; a < G; ++a) {
            const float4 q = cell_pos[p0 + ((mem >> a) & 1u ? a : lead)];
            ax[a] = -2.0f * q.x;
            ay[a] = -2.0f * q.y;
            az[a] = -2.0f * q.z;
            thr[a] = cut_scan - q.w;
        }
        // the runs as one list of chunks: lane r < 9 holds its run's chunks
        const int nck = (rend - rbeg + 31) >> 5;
        int upto = nck;  // chunks of the runs up to and with this one
#pragma unroll
        for (int o = 1; o < 16; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, upto, o);
            if (lane >= o) upto += u;
        }
        const int total = __shfl_sync(0xffffffffu, upto, 8);
        const unsigned lt = (1u << lane) - 1u;
        int nch = 0;
        for (int c0 = 0; c0 < total; c0 += 32) {
            // this lane's chunk: where it starts and which of its lanes exist
            int from = 0, left = 0;
#pragma unroll
            for (int r = 0; r < 9; ++r) {
                const int e = __shfl_sync(0xffffffffu, upto, r), n = __shfl_sync(0xffffffffu, nck, r);
                const int beg = __shfl_sync(0xffffffffu, rbeg, r), end = __shfl_sync(0xffffffffu, rend, r);
                const int at = c0 + lane - (e - n);
                if (at >= 0 && at < n) {
                    from = beg + 32 * at;
                    left = end - from;
                }
            }
            uint32_t keep[G];
#pragma unroll
            for (int a = 0; a < G; ++a) keep[a] = 0u;
            const int nin = min(32, total - c0);
            for (int c = 0; c < nin; c += 4) {  // four independent loads in flight
                float4 q[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) q[u] = cell_pos[__shfl_sync(0xffffffffu, from, c + u) + lane];
#pragma unroll
                for (int u = 0; u < 4; ++u)
#pragma unroll
                    for (int a = 0; a < G; ++a) {
                        const float t = fmaf(ax[a], q[u].x, fmaf(ay[a], q[u].y, fmaf(az[a], q[u].z, q[u].w)));
                        const uint32_t m = __ballot_sync(0xffffffffu, t < thr[a]);
                        keep[a] = lane == c + u ? m : keep[a];
                    }
            }
            // chunks with a candidate, compacted
            const uint32_t exist = left >= 32 ? 0xffffffffu : left > 0 ? (1u << left) - 1u : 0u;
            uint32_t any = 0u;
#pragma unroll
            for (int a = 0; a < G; ++a) any |= keep[a] &= exist;
            const unsigned some = __ballot_sync(0xffffffffu, any != 0u);
            const int at = nch + __popc(some & lt);
            if (any != 0u && at < NL_CHUNKS) {
                W.base[at] = from;
#pragma unroll
                for (int a = 0; a < G; ++a) W.bits[a][at] = keep[a];
            }
            nch += __popc(some);
        }
        __syncwarp();
#pragma unroll 1
        for (int a = 0; a < G; ++a) {
            if (!((mem >> a) & 1u)) continue;
            const int i = __shfl_sync(0xffffffffu, my_i, a);
            const double4 pi = ld_xyz(xyz, i);
            const double ri_pad = shorts ? prm64[4 * (size_t)i + 1] + reach_pad : 0.0;
            if (nch > NL_CHUNKS) {  // too many chunks to list: counted, then written, by FP64 scans
                int64_t off = 0;
                int c[4];
                nl_row_atom<0>(i, lane, g, xyz, rcut2, cell_of, cells, cell_atoms, prm64, reach_pad, excl_ptr,
                               excl_cols, excl_win, nl, c[0], c[1], c[2], c[3]);
                const int cnt = lane == 0 ? c[0] : lane == 1 ? c[1] : lane == 2 ? c[2] : c[3];
                if (take_rows(nl, s, cnt, lane, nkind, off, status)) {
                    set_rows(nl, i, cnt, lane, nkind, off);
                    __syncwarp();
                    nl_row_atom<1>(i, lane, g, xyz, rcut2, cell_of, cells, cell_atoms, prm64, reach_pad, excl_ptr,
                                   excl_cols, excl_win, nl, c[0], c[1], c[2], c[3]);
                }
                continue;
            }
            const float4 pf = cell_atom[p0 + a];
            const float rpad_f = (float)ri_pad;
            const uint4 ew = excl_window_of(excl_win, i);
            int cf = 0, cs = 0;  // this lane's entries: full | half << 16, short full | short half << 16
            int jmin = 0x7fffffff, jmax = -1;
            uint32_t *wf = nullptr, *wh = nullptr, *wsf = nullptr, *wsh = nullptr;
            // the candidates of chunks [b0, b1) into the stage: how many, or more than
            // NL_STAGE (and a useless stage) when they do not fit
            auto list = [&](int b0, int b1) {
                int n = 0;
                for (int b = b0; b < b1 && n <= NL_STAGE; b += 32) {
                    uint32_t m = b + lane < b1 ? W.bits[a][b + lane] : 0u;
                    const int32_t from = b + lane < b1 ? W.base[b + lane] : 0;
                    const int cnt = __popc(m);
                    int inc = cnt;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const int u = __shfl_up_sync(0xffffffffu, inc, o);
                        if (lane >= o) inc += u;
                    }
                    int at = n + inc - cnt;
                    n += __shfl_sync(0xffffffffu, inc, 31);
                    if (n <= NL_STAGE)
                        while (m) {
                            W.stage[at++] = (uint32_t)(from + __ffs(m) - 1);
                            m &= m - 1u;
                        }
                }
                __syncwarp();
                return n;
            };
            auto decide = [&](int n) {
#pragma unroll 2
                for (int t = lane; t < n; t += 32) {
                    const int k = (int)W.stage[t];
                    const int j = cell_atoms[k];
                    const float4 q = cell_atom[k];
                    const float dx = q.x - pf.x, dy = q.y - pf.y, dz = q.z - pf.z;
                    const float r2f = dx * dx + dy * dy + dz * dz;
                    uint32_t e = NL_DROPPED;
                    if (r2f < cut_hi && j != i) {
                        double r2 = -1.0;  // FP64 r², computed only when a test needs it
                        bool in = true, sh = false;
                        if (r2f > cut_lo) {
                            r2 = d2_of(pi, ld_xyz(xyz, j));
                            in = r2 < rcut2;
                        }
                        if (in && shorts) {
                            const float rf = rpad_f + q.w, rf2 = rf * rf;
                            if (r2f < rf2 - m2) {
                                sh = true;
                            } else if (r2f <= rf2 + m2) {
                                if (r2 < 0.0) r2 = d2_of(pi, ld_xyz(xyz, j));
                                const double reach = ri_pad + prm64[4 * (size_t)j + 1];
                                sh = r2 < reach * reach;
                            }
                        }
                        if (in) {
                            e = (uint32_t)j |
                                (excluded_w(excl_win, ew, excl_ptr, excl_cols, i, j) ? ALMA_EXCL_BIT : 0u) |
                                (sh ? NL_SHORT_BIT : 0u);
                            const int up = j > i ? 0x10001 : 1;
                            cf += up;
                            cs += sh ? up : 0;
                            jmin = min(jmin, j);
                            jmax = max(jmax, j);
                        }
                    }
                    W.stage[t] = e;
                }
            };
            auto place = [&] {
                int64_t off = 0;
                cf = __reduce_add_sync(0xffffffffu, cf);
                cs = __reduce_add_sync(0xffffffffu, cs);
                const int cnt = lane == 0 ? cf & 0xffff : lane == 1 ? cf >> 16 : lane == 2 ? cs & 0xffff : cs >> 16;
                if (!take_rows(nl, s, cnt, lane, nkind, off, status)) return false;
                set_rows(nl, i, cnt, lane, nkind, off);
                if (lane == 0) *reinterpret_cast<double4 *>(nl.ref_xyz + 4 * (size_t)i) = pi;
                if (nl.full_span != nullptr) {
                    jmin = __reduce_min_sync(0xffffffffu, jmin);
                    jmax = __reduce_max_sync(0xffffffffu, jmax);
                    if (lane == 0) {
                        nl.full_span[2 * (size_t)i] = jmin;
                        nl.full_span[2 * (size_t)i + 1] = jmax;
                    }
                }
                wf = nl.full_cols + __shfl_sync(0xffffffffu, off, 0);
                wh = nl.half_cols + __shfl_sync(0xffffffffu, off, 1);
                wsf = shorts ? nl.sfull_cols + __shfl_sync(0xffffffffu, off, 2) : nullptr;
                wsh = shorts ? nl.shalf_cols + __shfl_sync(0xffffffffu, off, 3) : nullptr;
                return true;
            };
            auto write = [&](int n) {
                for (int t0 = 0; t0 < n; t0 += 32) {
                    const uint32_t st = t0 + lane < n ? W.stage[t0 + lane] : NL_DROPPED;
                    const bool v = st != NL_DROPPED;
                    const bool hf = v && (int)(st & (ALMA_IDX_MASK & ~NL_SHORT_BIT)) > i;
                    const unsigned mf = __ballot_sync(0xffffffffu, v), mh = __ballot_sync(0xffffffffu, hf);
                    const uint32_t e = st & ~NL_SHORT_BIT;
                    if (v) wf[__popc(mf & lt)] = e;
                    if (hf) wh[__popc(mh & lt)] = e;
                    wf += __popc(mf);
                    wh += __popc(mh);
                    if (shorts) {
                        const bool sh = v && (st & NL_SHORT_BIT);
                        const unsigned ms = __ballot_sync(0xffffffffu, sh), msh = ms & mh;
                        if (sh) {
                            wsf[__popc(ms & lt)] = e;
                            if (hf) wsh[__popc(msh & lt)] = e;
                        }
                        wsf += __popc(ms);
                        wsh += __popc(msh);
                    }
                }
                __syncwarp();  // the stage is the next part's
            };
            const int n = list(0, nch);
            if (n > NL_STAGE) {
                // too long for the stage: 32 chunks (1,024 candidates at most) at a
                // time, once to be counted and again to be written.  48 chains of
                // 4,962 atoms scaled to 0.9, where one row in six is that long:
                // 2,719 us, 3,955 with FP64 scans of the 27 cells for those.
                const int parts = (nch + 31) >> 5;
#pragma unroll 1
                for (int p = 0; p < 2 * parts; ++p) {
                    if (p == parts && !place()) break;
                    const int b = 32 * (p < parts ? p : p - parts);
                    const int part = list(b, min(nch, b + 32));
                    decide(part);
                    if (p >= parts) write(part);
                    __syncwarp();
                }
                continue;
            }
            decide(n);
            if (place()) write(n);
            else __syncwarp();
        }
        __syncwarp();  // the masks and the stage are the next atoms'
    }
}

// Exclusion windows (alma_excl_window): thread per atom over its CSR row
// (partners j > i); each pair sets its bit in both atoms' windows, or the
// far flag (bit 64) of both when j - i >= EXCL_WIN.
__global__ void excl_window_kernel(const int64_t *__restrict__ excl_ptr, const int32_t *__restrict__ excl_cols,
                                   int natoms, uint32_t *__restrict__ win) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= natoms) return;
    for (int64_t k = excl_ptr[i]; k < excl_ptr[i + 1]; ++k) {
        const int j = excl_cols[k];
        if (j < 0 || j >= natoms || j == i) continue;
        const int d = j - i;
        if (d > -EXCL_WIN && d < EXCL_WIN) {
            const unsigned bi = (unsigned)(d + EXCL_WIN), bj = (unsigned)(EXCL_WIN - d);
            atomicOr(&win[4 * (size_t)i + (bi >> 5)], 1u << (bi & 31u));
            atomicOr(&win[4 * (size_t)j + (bj >> 5)], 1u << (bj & 31u));
        } else {
            atomicOr(&win[4 * (size_t)i + 2], 1u);
            atomicOr(&win[4 * (size_t)j + 2], 1u);
        }
    }
}

}  // namespace alma

using namespace alma;

extern "C" int alma_excl_window(const int64_t *excl_ptr, const int32_t *excl_cols, int32_t natoms, uint32_t *win,
                                void *stream) {
    if (natoms < 0 || (natoms > 0 && (!excl_ptr || !excl_cols || !win)))
        return alma_set_error(ALMA_EINVAL, "alma_excl_window: bad arguments");
    if (natoms == 0) return ALMA_OK;
    cudaStream_t st = (cudaStream_t)stream;
    ALMA_CUDA_TRY(cudaMemsetAsync(win, 0, sizeof(uint32_t) * 4 * (size_t)natoms, st));
    excl_window_kernel<<<(natoms + 255) / 256, 256, 0, st>>>(excl_ptr, excl_cols, natoms, win);
    ALMA_LAUNCH_CHECK("alma_excl_window");
    return ALMA_OK;
}

extern "C" size_t alma_nl_workspace_bytes(int32_t nsys, int32_t natoms, int64_t max_cells) {
    return carve(nullptr, nullptr, nsys, natoms, max_cells);
}

extern "C" int alma_nl_build(const AlmaBatch *b, const AlmaTopo *t, AlmaNL *nl, const AlmaParams *p,
                             const uint8_t *sys_mask, void *workspace, int64_t max_cells, void *stream) {
    if (!b || !nl || !workspace || b->nsys <= 0 || b->natoms < 0 || max_cells <= 0)
        return alma_set_error(ALMA_EINVAL, "alma_nl_build: bad arguments");
    if (b->natoms >= (1 << 30))  // the build stages a flag in bit 30 of each entry
        return alma_set_error(ALMA_EINVAL, "alma_nl_build: at most 2^30 - 1 atoms");
    if (!nl->full_ptr || !nl->full_len || !nl->half_ptr || !nl->half_len || !nl->full_base || !nl->half_base ||
        !nl->ref_xyz || !nl->need || !b->xyz || !b->atom_off)
        return alma_set_error(ALMA_EINVAL, "alma_nl_build: null buffer");
    if (nl->sfull_cols && (!nl->sfull_ptr || !nl->sfull_len || !nl->sfull_base || !nl->shalf_ptr || !nl->shalf_len ||
                           !nl->shalf_cols || !nl->shalf_base || !b->prm64))
        return alma_set_error(ALMA_EINVAL, "alma_nl_build: incomplete short rows");
    AlmaParams pref;
    if (!p) {
        alma_params_reference(&pref);
        p = &pref;
    }
    // SASA reach R*_i + R*_j + 2 probe, plus the skin (both atoms may each
    // drift half the skin before a rebuild).
    // A 1e-6 A margin keeps rounding at the boundary on the safe side.
    const double reach_pad = 2.0 * p->probe_r + 2.0 * sqrt(p->half_skin2) + 1e-6;
    cudaStream_t st = (cudaStream_t)stream;
    const int nsys = b->nsys, natoms = b->natoms;
    NLWork w;
    carve(&w, (char *)workspace, nsys, natoms, max_cells);
    if (natoms == 0) return ALMA_OK;
    ALMA_CUDA_TRY(cudaMemsetAsync(w.total_cells, 0, sizeof(unsigned long long), st));
    const double rcut2 = (12.0 + 2.0) * (12.0 + 2.0);
    // Four atoms per thread, up to 8 CTAs (the portable cluster): a cluster
    // barrier costs as much as a few more atoms per thread (1,089 atoms: 7 us
    // with one CTA, 10.5 with two; 200 x 4.9k atoms: 60 us, 119 at two atoms).
    const int avg = natoms / nsys, unit = 4 * CELLS_THREADS;
    const int cl = avg <= unit ? 1 : avg <= 2 * unit ? 2 : avg <= 4 * unit ? 4 : 8;
    auto cells = cl == 1 ? nl_cells_kernel<1> : cl == 2 ? nl_cells_kernel<2> : cl == 4 ? nl_cells_kernel<4>
                                                                                     : nl_cells_kernel<8>;
    ALMA_CUDA_TRY(alma_launch_cluster(cells, (unsigned)nsys * (unsigned)cl, CELLS_THREADS, (unsigned)cl, (size_t)0,
                                      st, b->atom_off, sys_mask, b->xyz, rcut2, max_cells, w.grid, w.total_cells,
                                      w.cell_of, w.cell_end, w.scattered, nl->need, b->status));
    nl_order_kernel<<<(natoms + 255) / 256, 256, 0, st>>>(b->atom_off, nsys, natoms, sys_mask, w.grid, w.cell_of,
                                                          w.cell_end, w.scattered, b->xyz, b->prm64, w.cell_atoms,
                                                          w.cell_pos, w.cell_atom);
    const int64_t *ep = t ? t->excl_ptr : nullptr;
    const int32_t *ec = t ? t->excl_cols : nullptr;
    const uint32_t *ew = t && t->excl_ptr ? t->excl_win : nullptr;
    // Two atoms per warp read each candidate once for both; below about two
    // waves of one-atom warps the chip has room for the shorter chains (16k
    // atoms: 94 us with one, 95 with two; 24k: 157 and 150; 32k: 174 and 166; 65k:
    // 481 and 431).
    auto rows = [&](auto kfn, int per_warp) {
        const int per_block = per_warp * NL_WARPS;
        kfn<<<(natoms + per_block - 1) / per_block, NL_WARPS * 32, 0, st>>>(
            b->atom_off, nsys, natoms, sys_mask, b->xyz, rcut2, w.grid, w.cell_of, w.cell_end, w.cell_atoms,
            w.cell_pos, w.cell_atom, b->prm64, reach_pad, ep, ec, ew, *nl, b->status);
    };
    if (natoms >= 24000) rows(nl_rows_kernel<2>, 2);
    else rows(nl_rows_kernel<1>, 1);
    ALMA_LAUNCH_CHECK_N("alma_nl_build", 3);
    return ALMA_OK;
}
