// pgmpm_hashgrid.cu -- spatial hash grid for particle neighbourhoods on the
// GPU: the structure of physgrad::sparse::SpatialHashGrid<float, uint32_t>
// (src/sparse_data_structures.h:44-296; used by the FSI coupling,
// src/fsi_coupling.h:72), with its build and neighbour query as kernels.
//
//   cell id    morton(c) % total_cells, c = the cell coordinates of a point,
//              truncated to uint32 and clamped to the resolution (the
//              reference's getCellID, :143-151, Morton code :121-131)
//   build      per-cell counts (a histogram of the cell ids), starts (their
//              exclusive scan) and a stable sort of (cell id, particle index)
//              pairs (the existing LSD radix sort): the reference's count /
//              exclusive scan / stable fill (:155-190) give the same arrays
//   neighbours for a query point, every particle stored in the cells of the
//              (2 ceil(r / cell) + 1)^3 block around its cell, in the
//              reference's order (x outer, z inner; a cell's particles by
//              index), with no distance test -- as getNeighbors (:206-240),
//              which computes radius^2 but does not use it.  Two passes: a
//              count (thread per query), a scan into offsets, then the fill
//              (8 lanes per query, so each list is written contiguously).
//
// Float arithmetic is IEEE single (no contraction), so cell ids match the
// reference's host code bit for bit.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>

#include "pgmpm_hashgrid.cuh"
#include "pgmpm_solver_impl.h"

using namespace pgmpm;

struct pgmpm_hashgrid_s {
    int device = 0;
    float cell = 0.f;
    float dmin[3] = {0.f, 0.f, 0.f};
    uint32_t res[3] = {0, 0, 0};
    uint32_t total = 0;
    int key_bits = 1;
    int64_t max_particles = 0;
    int64_t n = 0;  // particles of the last build
    bool built = false;
    // Buffers of a size known at creation, in one allocation (every one of a
    // megabyte and more takes 0.34 ms; see layout())
    DevBuf mem;
    uint32_t *counts = nullptr, *starts = nullptr;  // per cell
    uint32_t* cell_ids = nullptr;                   // per particle: cell id (particle order)
    // sort buffers; between builds va keeps the sorted particle indices, ka
    // holds the queries' cells, and kb and vb, one stretch, the index in grid order
    uint32_t *ka = nullptr, *va = nullptr, *kb = nullptr, *vb = nullptr, *scratch = nullptr;
    unsigned long long* stats = nullptr;
    int64_t* scan = nullptr;    // block sums of a scan over cells or up to max_particles queries
    int64_t* result = nullptr;  // [0] length of a query set's lists, [1] entries of the index in grid order
    uint32_t* qcount = nullptr; // counts of up to max_particles queries (null: qlarge)
    // dense queries (cells in grid order, x outer, z inner; null: hashed queries
    // only): z stretches and block sums for the last half width, and first[] of
    // the cells' buckets
    uint2* grid_rows = nullptr;
    uint32_t *grid_sum = nullptr, *grid_first = nullptr;
    DevBuf pos_stage, qstage, qout_stage, off_stage;  // host arrays on the device
    DevBuf qlarge;      // counts, cells and block sums of more than max_particles queries
    DevBuf grid_index;  // the index in grid order where kb and vb are too short for it
    int64_t index_need = 0;   // entries that did not fit
    bool grid_ready = false;  // grid_first and the index hold the last build's
    int64_t sum_src = -1;     // grid_rows and grid_sum hold the last build's for this half width

    int64_t stride() const { return (std::max<int64_t>(max_particles, 1) + 63) & ~63ll; }
    uint32_t* index() const { return grid_index.p ? grid_index.as<uint32_t>() : kb; }
    int64_t index_capacity() const { return grid_index.p ? (int64_t)(grid_index.bytes / sizeof(uint32_t)) : 2 * stride(); }
    size_t layout(bool dense);  // places the buffers in mem (if it is allocated); their bytes together
};

namespace {

constexpr int HG_T = 256;

// cell id per particle, and the per-cell counts (one atomic per particle:
// input order is arbitrary, so a warp's particles rarely share a cell and
// aggregating them over the warp cost more than it saved)
__global__ void k_hg_cells(HGDev G, const float* __restrict__ pos, int64_t n, uint32_t* __restrict__ cell_ids,
                           uint32_t* __restrict__ counts) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint32_t c[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) c[a] = min(hg_coord(pos[3 * i + a], G.dmin[a], G.cell), G.res[a] - 1u);
    const uint32_t id = hg_mod(hg_morton(c[0], c[1], c[2]), G);
    cell_ids[i] = id;
    atomicAdd(&counts[id], 1u);
}

// Count pass, one thread per query: the block's cells in nested loops (the
// reference's order does not matter for a sum)
__global__ void k_hg_qcount(HGDev G, const float* __restrict__ q, int64_t nq, uint32_t src,
                            const uint32_t* __restrict__ counts, uint32_t* __restrict__ qcount) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nq) return;
    uint32_t c[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) c[a] = hg_coord(q[3 * i + a], G.dmin[a], G.cell);
    uint32_t k = 0;
    for (uint32_t dx = 0; dx <= 2 * src; ++dx) {
        const uint32_t gx = c[0] + dx - src;  // uint32 wrap: below 0 fails the range test
        if (gx >= G.res[0]) continue;
        for (uint32_t dy = 0; dy <= 2 * src; ++dy) {
            const uint32_t gy = c[1] + dy - src;
            if (gy >= G.res[1]) continue;
            for (uint32_t dz = 0; dz <= 2 * src; ++dz) {
                const uint32_t gz = c[2] + dz - src;
                if (gz >= G.res[2]) continue;
                k += counts[hg_mod(hg_morton(gx, gy, gz), G)];
            }
        }
    }
    qcount[i] = k;
}

// Fill pass, HG_FG lanes per query: they take the block's cells in the
// reference's order (linear index t = (dx (2s+1) + dy) (2s+1) + dz), HG_FG at
// a time, give each cell its place by a scan over the lanes and copy the
// cell's particles, so a query's list is written into one contiguous stretch
// by its lanes together.
constexpr int HG_FG = 8;  // lanes per query in the fill (4 queries per warp; 4 lanes and 32 were slower)
__global__ void k_hg_qfill(HGDev G, const float* __restrict__ q, int64_t nq, uint32_t src,
                           const uint32_t* __restrict__ counts, const uint32_t* __restrict__ starts,
                           const uint32_t* __restrict__ sorted_index, const int64_t* __restrict__ offsets,
                           uint32_t* __restrict__ out) {
    __shared__ uint32_t tab[HG_TAB];
    const uint32_t w = 2 * src + 1, ncell = w * w * w;
    hg_fill_table(tab, ncell, w);
    const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / HG_FG;
    const int lane = threadIdx.x & 31, sub = lane % HG_FG;
    const uint32_t gmask = ((1u << HG_FG) - 1u) << (lane - sub);  // this query's lanes
    if (i >= nq) return;  // a query's lanes leave together
    uint32_t c[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) c[a] = hg_coord(q[3 * i + a], G.dmin[a], G.cell);
    int64_t o = offsets[i];
    for (uint32_t t0 = 0; t0 < ncell; t0 += HG_FG) {
        const uint32_t t = t0 + sub;
        uint32_t id = 0, k = 0, s0 = 0;
        if (t < ncell && hg_cell_of(G, c, src, w, ncell, tab, t, id)) {
            k = counts[id];
            s0 = starts[id];
        }
        uint32_t x = k;  // inclusive scan of the counts over the query's lanes
#pragma unroll
        for (int d = 1; d < HG_FG; d <<= 1) {
            const uint32_t y = __shfl_up_sync(gmask, x, d, HG_FG);
            if (sub >= d) x += y;
        }
        const uint32_t kmax = __reduce_max_sync(gmask, k);
        if (kmax < 2 * HG_FG) {
            // short cells: each lane copies its own cell's entries
            const int64_t base = o + (x - k);
            for (uint32_t j = 0; j < k; ++j) out[base + j] = sorted_index[s0 + j];
        } else {
            // long cells: the query's lanes copy each cell together, so the
            // list is written (and the sorted index read) in runs
#pragma unroll 1
            for (int m = 0; m < HG_FG; ++m) {
                const uint32_t km = __shfl_sync(gmask, k, m, HG_FG);
                const uint32_t sm = __shfl_sync(gmask, s0, m, HG_FG);
                const int64_t bm = o + (__shfl_sync(gmask, x, m, HG_FG) - km);
                for (uint32_t j = (uint32_t)sub; j < km; j += HG_FG) out[bm + j] = sorted_index[sm + j];
            }
        }
        o += __shfl_sync(gmask, x, HG_FG - 1, HG_FG);
    }
}

// Exclusive scan of n uint32 counts into out[0..n] (out[n] = total, where
// asked for): per-block sums, one block scanning the sums, then each block's
// scan plus its carry.  A warp takes ROWS rows of 32 counts, every access a full
// line: 4 rows for many counts (2 M: sums 10 -> 3.9 us, apply 11.4 -> 7.7 us
// against one count per thread), one where latency counts (apply of 1 to 20,000
// counts 2.0-2.2 us, 2.9-3.2 with four).
constexpr int SCAN_T = 1024;
constexpr int64_t SCAN_FEW = (int64_t)1 << 18;  // most counts for one row
constexpr int scan_rows(int64_t n) { return n <= SCAN_FEW ? 1 : 4; }
constexpr int64_t scan_blocks(int64_t n) {
    return (n + SCAN_T * scan_rows(n) - 1) / (SCAN_T * scan_rows(n));
}
// block sums of any scan of up to n counts
constexpr int64_t scan_words(int64_t n) {
    return n <= SCAN_FEW ? scan_blocks(n) : scan_blocks(n) > scan_blocks(SCAN_FEW) ? scan_blocks(n) : scan_blocks(SCAN_FEW);
}
__device__ __forceinline__ int64_t warp_incl_scan(int64_t x, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int64_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= o) x += y;
    }
    return x;
}
__device__ __forceinline__ int64_t block_incl_scan(int64_t x, int64_t* sh) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    x = warp_incl_scan(x, lane);
    if (lane == 31) sh[warp] = x;
    __syncthreads();
    if (warp == 0) sh[lane] = warp_incl_scan(lane < SCAN_T / 32 ? sh[lane] : 0, lane);
    __syncthreads();
    const int64_t r = x + (warp ? sh[warp - 1] : 0);
    __syncthreads();
    return r;
}
template <int ROWS>
__global__ void __launch_bounds__(SCAN_T) k_scan_sums(const uint32_t* __restrict__ in, int64_t n,
                                                      int64_t* __restrict__ bsum) {
    __shared__ int64_t sh[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int64_t s = 0;
#pragma unroll
    for (int k = 0; k < ROWS; ++k) {
        const int64_t i = (int64_t)blockIdx.x * (SCAN_T * ROWS) + k * SCAN_T + threadIdx.x;
        s += i < n ? in[i] : 0u;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xFFFFFFFFu, s, o);
    if (lane == 0) sh[warp] = s;
    __syncthreads();
    if (warp == 0) {
        s = sh[lane];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xFFFFFFFFu, s, o);
        if (lane == 0) bsum[blockIdx.x] = s;
    }
}
__global__ void __launch_bounds__(SCAN_T) k_scan_carry(int64_t* __restrict__ bsum, int64_t nb) {
    __shared__ int64_t sh[32];
    __shared__ int64_t s_tot;
    int64_t carry = 0;
    for (int64_t b0 = 0; b0 < nb; b0 += SCAN_T) {
        const int64_t i = b0 + threadIdx.x;
        const int64_t v = i < nb ? bsum[i] : 0;
        const int64_t r = block_incl_scan(v, sh);
        if (i < nb) bsum[i] = carry + r - v;  // exclusive, over all blocks so far
        if (threadIdx.x == SCAN_T - 1) s_tot = r;
        __syncthreads();
        carry += s_tot;
        __syncthreads();
    }
}
// OutT: int64 query offsets or uint32 cell starts
// (TOTAL: out[n] too, and the total in 64 bits where asked for)
template <int ROWS, class OutT, bool TOTAL>
__global__ void __launch_bounds__(SCAN_T) k_scan_apply(const uint32_t* __restrict__ in, int64_t n,
                                                       const int64_t* __restrict__ bsum, OutT* __restrict__ out,
                                                       int64_t* __restrict__ total) {
    __shared__ int64_t sh[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t base = (int64_t)blockIdx.x * (SCAN_T * ROWS) + warp * (32 * ROWS) + lane;
    int64_t v[ROWS], x[ROWS], run = 0;
#pragma unroll
    for (int k = 0; k < ROWS; ++k) v[k] = base + 32 * k < n ? in[base + 32 * k] : 0u;
#pragma unroll
    for (int k = 0; k < ROWS; ++k) {  // inclusive over the warp's rows so far
        x[k] = run + warp_incl_scan(v[k], lane);
        run = __shfl_sync(0xFFFFFFFFu, x[k], 31);
    }
    if (lane == 0) sh[warp] = run;
    __syncthreads();
    if (warp == 0) sh[lane] = warp_incl_scan(sh[lane], lane);
    __syncthreads();
    const int64_t before = bsum[blockIdx.x] + (warp ? sh[warp - 1] : 0);
#pragma unroll
    for (int k = 0; k < ROWS; ++k) {
        const int64_t i = base + 32 * k;
        if (i < n) out[i] = (OutT)(before + x[k] - v[k]);
        if (TOTAL && i == n - 1) {
            out[n] = (OutT)(before + x[k]);
            if (total) *total = before + x[k];
        }
    }
}

// (out[n] and *total where TOTAL; n > 0, bsum of scan_words(n))
template <class OutT, bool TOTAL>
cudaError_t scan_counts(const uint32_t* in, int64_t n, int64_t* bsum, OutT* out, int64_t* total, cudaStream_t st) {
    const int nb = (int)scan_blocks(n);
    const bool few = scan_rows(n) == 1;
    if (few)
        k_scan_sums<1><<<nb, SCAN_T, 0, st>>>(in, n, bsum);
    else
        k_scan_sums<4><<<nb, SCAN_T, 0, st>>>(in, n, bsum);
    k_scan_carry<<<1, SCAN_T, 0, st>>>(bsum, nb);
    if (few)
        k_scan_apply<1, OutT, TOTAL><<<nb, SCAN_T, 0, st>>>(in, n, bsum, out, total);
    else
        k_scan_apply<4, OutT, TOTAL><<<nb, SCAN_T, 0, st>>>(in, n, bsum, out, total);
    return cudaGetLastError();
}

// ------------------------------------------------------ dense query sets
// When the queries are at least 1/4 of the cells and have 2^19 cells to look up
// (HG_DENSE_CELLS, HG_DENSE_WORK), the index is first laid out again in grid order (x outer, z inner): every cell's bucket, one after the
// other, so that the 2s+1 cells of a query's block along z are one stretch of
// it and no query hashes anything:
//   k_hg_grid    (start, count) of every cell, scanned into the stretches
//   k_hg_expand  the buckets in grid order (those that several cells hash to are
//                repeated: up to 1.8 times the particles for uniform clouds in a
//                cube of cells, none where its edge is a power of two)
//   k_hg_rows    each cell's stretch of 2s+1 cells along z
//   k_hg_blocks  and the particles of its whole block, once per cell instead of
//                once per query
//   k_hg_dcount  per query: its cell's block sum
//   k_hg_dfill   27 lanes for three queries (or a warp per query): a lane reads
//                one stretch, the lanes then take the lists' entries in turn
//                (hg_walk), so that lists are written in full lines
// Bound by scattered L1/L2 accesses.  2 M queries over 2 M cells of one
// particle each (27 cells per query): count and fill 168 + 496 us with the
// hashed kernels (27 scattered 4-byte reads a query and pass, entries copied
// cell by cell), 15 + 228 us here and 64 us for the layout (380 us for the fill
// with one query per warp and a lane per cell).
constexpr uint32_t HG_OUTSIDE = 0xFFFFFFFFu;  // qcell: the query is outside the grid

__global__ void k_hg_grid(HGDev G, const uint32_t* __restrict__ counts, const uint32_t* __restrict__ starts,
                          uint32_t* __restrict__ ccount, uint32_t* __restrict__ cstart) {
    const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= G.total) return;
    const uint32_t z = c % G.res[2], xy = c / G.res[2], y = xy % G.res[1], x = xy / G.res[1];
    const uint32_t id = hg_mod(hg_morton(x, y, z), G);
    ccount[c] = counts[id];
    cstart[c] = starts[id];
}
// first[c] .. first[c + 1]: cell c's bucket in grid order.  Nothing is written
// when the entries exceed capacity (first may then have wrapped, too).
__global__ void k_hg_expand(uint32_t total, const uint32_t* __restrict__ first, const uint32_t* __restrict__ cstart,
                            const uint32_t* __restrict__ sorted_index, const int64_t* __restrict__ entries,
                            int64_t capacity, uint32_t* __restrict__ out) {
    const int64_t have = *entries;  // (read along with first)
    // warps copy their 32 cells' buckets together: one stretch of out
    const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t f = c < total ? first[c] : 0u, k = c < total ? first[c + 1] - f : 0u;
    const int lane = threadIdx.x & 31;
    if (have > capacity) return;
    uint32_t* dst = out + __shfl_sync(0xFFFFFFFFu, f, 0);
    hg_walk(c < total ? cstart[c] : 0u, k, lane, [&](bool valid, uint32_t e, uint32_t pos) {
        if (valid) dst[e] = __ldg(&sorted_index[pos]);
    });
}
__global__ void k_hg_rows(HGDev G, uint32_t src, const uint32_t* __restrict__ first, uint2* __restrict__ rows) {
    const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= G.total) return;
    const uint32_t z = c % G.res[2], row = c - z;
    const uint32_t f = first[row + (z > src ? z - src : 0u)];
    rows[c] = make_uint2(f, first[row + min(z + src, G.res[2] - 1u) + 1u] - f);
}
__global__ void k_hg_blocks(HGDev G, uint32_t src, const uint2* __restrict__ rows, uint32_t* __restrict__ sums) {
    const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= G.total) return;
    const uint32_t z = c % G.res[2], xy = c / G.res[2], y = xy % G.res[1], x = xy / G.res[1];
    const uint32_t x0 = x > src ? x - src : 0u, x1 = min(x + src, G.res[0] - 1u);
    const uint32_t y0 = y > src ? y - src : 0u, y1 = min(y + src, G.res[1] - 1u);
    uint32_t k = 0;
    for (uint32_t i = x0; i <= x1; ++i)
        for (uint32_t j = y0; j <= y1; ++j) k += rows[(i * G.res[1] + j) * G.res[2] + z].y;
    sums[c] = k;
}
__global__ void k_hg_dcount(HGDev G, const float* __restrict__ q, int64_t nq, uint32_t src,
                            const uint32_t* __restrict__ first, const uint32_t* __restrict__ sums,
                            uint32_t* __restrict__ qcount, uint32_t* __restrict__ qcell) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nq) return;
    uint32_t c[3];
    bool in = true;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        c[a] = hg_coord(q[3 * i + a], G.dmin[a], G.cell);
        in = in && c[a] < G.res[a];
    }
    const uint32_t lin = (c[0] * G.res[1] + c[1]) * G.res[2] + c[2];
    uint32_t k = 0;
    if (in)
        k = sums[lin];
    else
        for (uint32_t dx = 0; dx <= 2 * src; ++dx)
            for (uint32_t dy = 0; dy <= 2 * src; ++dy) k += hg_row(G, c, src, dx, dy, first).y;
    qcount[i] = k;
    qcell[i] = in ? lin : HG_OUTSIDE;
}
// Nothing is written when the lists (offsets[nq] entries) exceed capacity, or
// the index in grid order was not written.
// QW: queries a warp takes together; their lists are one stretch of out, and
// (2 src + 1)^2 QW <= 32 stretches come from one read per lane.  QW = 1 also
// takes wider blocks, 32 stretches at a time.
template <int QW>
__global__ void __launch_bounds__(HG_T) k_hg_dfill(HGDev G, const float* __restrict__ q, int64_t nq, uint32_t src,
                                                   const uint32_t* __restrict__ first, const uint2* __restrict__ rows,
                                                   const uint32_t* __restrict__ index,
                                                   const uint32_t* __restrict__ qcell,
                                                   const int64_t* __restrict__ entries, int64_t index_capacity,
                                                   const int64_t* __restrict__ offsets, int64_t capacity,
                                                   uint32_t* __restrict__ out) {
    const int64_t length = offsets[nq], have = *entries;
    if (length > capacity || have > index_capacity) return;
    const uint32_t w = 2 * src + 1, nrow = w * w;
    const int lane = threadIdx.x & 31;
    const uint32_t mine = QW > 1 ? lane / nrow : 0u;  // this lane's query of the warp's, and its row of it
    const uint32_t r1 = QW > 1 ? lane % nrow : (uint32_t)lane;
    const int64_t step = (int64_t)gridDim.x * (HG_T / 32) * QW;
    for (int64_t i0 = ((int64_t)blockIdx.x * (HG_T / 32) + (threadIdx.x >> 5)) * QW; i0 < nq; i0 += step) {
        uint32_t* dst = out + offsets[i0];
        const int64_t i = i0 + mine;
        const uint32_t lin = mine < (uint32_t)QW && i < nq ? qcell[i] : HG_OUTSIDE;
        for (uint32_t r0 = 0; r0 < nrow; r0 += 32) {
            const uint32_t r = r0 + r1;
            uint2 seg = make_uint2(0u, 0u);
            if (r < nrow && mine < (uint32_t)QW && i < nq) {
                const uint32_t dx = r / w, dy = r % w;
                if (lin != HG_OUTSIDE) {
                    const uint32_t xy = lin / G.res[2], y = xy % G.res[1] + dy - src, x = xy / G.res[1] + dx - src;
                    if (x < G.res[0] && y < G.res[1])
                        seg = __ldg(&rows[lin + ((dx - src) * G.res[1] + (dy - src)) * G.res[2]]);
                } else {
                    uint32_t c[3];
#pragma unroll
                    for (int a = 0; a < 3; ++a) c[a] = hg_coord(q[3 * i + a], G.dmin[a], G.cell);
                    seg = hg_row(G, c, src, dx, dy, first);
                }
            }
            dst += hg_walk(seg.x, seg.y, lane, [&](bool valid, uint32_t e, uint32_t pos) {
                if (valid) dst[e] = __ldg(&index[pos]);
            });
            if (QW > 1) break;
        }
    }
}

__global__ void k_hg_stats(const uint32_t* __restrict__ counts, uint32_t total,
                           unsigned long long* __restrict__ st) {  // occupied, max, particles
    uint32_t occ = 0, mx = 0;
    unsigned long long sum = 0;
    for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < total; c += gridDim.x * blockDim.x) {
        const uint32_t k = counts[c];
        occ += k > 0;
        mx = max(mx, k);
        sum += k;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        occ += __shfl_down_sync(0xFFFFFFFFu, occ, o);
        mx = max(mx, __shfl_down_sync(0xFFFFFFFFu, mx, o));
        sum += __shfl_down_sync(0xFFFFFFFFu, sum, o);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&st[0], (unsigned long long)occ);
        atomicMax(&st[1], (unsigned long long)mx);
        atomicAdd(&st[2], sum);
    }
}

HGDev dev_of(const pgmpm_hashgrid_s* g) {
    HGDev d;
    d.cell = g->cell;
    for (int a = 0; a < 3; ++a) {
        d.dmin[a] = g->dmin[a];
        d.res[a] = g->res[a];
    }
    d.total = g->total;
    d.total_m = ~0ull / g->total + 1ull;  // wraps to 0 for total = 1, where every remainder is 0
    return d;
}

int blocks_of(int64_t n, int t) { return (int)std::max<int64_t>(1, (n + t - 1) / t); }

// copies nfloat floats from host (or takes the device pointer) into stage
const float* staged(DevBuf& stage, const float* p, int64_t nfloat, int32_t kind, cudaStream_t st, int& rc) {
    rc = PGMPM_OK;
    if (kind == PGMPM_PTR_DEVICE) return p;
    if (stage.ensure(sizeof(float) * std::max<int64_t>(nfloat, 1)) != cudaSuccess) {
        rc = fail(PGMPM_ERR_OOM, "hashgrid: staging allocation failed");
        return nullptr;
    }
    if (nfloat && cudaMemcpyAsync(stage.p, p, sizeof(float) * nfloat, cudaMemcpyHostToDevice, st) != cudaSuccess) {
        rc = fail(PGMPM_ERR_CUDA, "hashgrid: host copy failed");
        return nullptr;
    }
    return stage.as<float>();
}

// Where the grid-order tables pay: laying them out costs 30 ps per cell (2 M
// cells), and a hashed query of 27 cells 0.2 ns more than a dense one; and their
// seven launches cost about as much as 2^19 cell lookups of the queries.  First
// query of a build, hashed and dense: 500 queries of 27 cells 61 and 80 us, 8,000
// 68 and 78, 20,000 76 and 76, 5,000 of 125 cells 115 and 81, 60,000 of 27 88 and
// 82, 200,000 119 and 103, 2 M 1075 and 368 us.
constexpr int64_t HG_DENSE_CELLS = 4;         // most cells per query
constexpr int64_t HG_DENSE_WORK = 1ll << 19;  // least cells of all queries' blocks together

// The grid-order tables of the last build for blocks of half width src (kept
// until the next build).  1: ready, unless result[1] shows more entries than
// the index holds; 0: the memory for it is not to be had; < 0: an error.
int dense_tables(pgmpm_hashgrid_s* g, const HGDev& G, uint32_t src, cudaStream_t st) {
    if (g->index_need > g->index_capacity()) {
        const size_t words = (size_t)g->index_need + (size_t)g->index_need / 4;
        if (g->grid_index.alloc(sizeof(uint32_t) * words) != cudaSuccess) {
            cudaGetLastError();  // clear the failed allocation
            return 0;
        }
        g->grid_ready = false;
    }
    const int nb = blocks_of((int64_t)g->total, HG_T);
    if (!g->grid_ready) {
        uint32_t* cstart = reinterpret_cast<uint32_t*>(g->grid_rows);  // until k_hg_rows writes it
        k_hg_grid<<<nb, HG_T, 0, st>>>(G, g->counts, g->starts, g->grid_sum, cstart);
        CK(exclusive_scan(g->grid_sum, (int64_t)g->total, g->scan, g->grid_first, st, g->result + 1));
        k_hg_expand<<<nb, HG_T, 0, st>>>(g->total, g->grid_first, cstart, g->va, g->result + 1, g->index_capacity(),
                                         g->index());
    }
    if (!g->grid_ready || g->sum_src != (int64_t)src) {
        k_hg_rows<<<nb, HG_T, 0, st>>>(G, src, g->grid_first, g->grid_rows);
        k_hg_blocks<<<nb, HG_T, 0, st>>>(G, src, g->grid_rows, g->grid_sum);
    }
    CK(cudaGetLastError());
    g->grid_ready = true;
    g->sum_src = src;
    return 1;
}

}  // namespace

namespace pgmpm {
size_t exclusive_scan_bytes(int64_t n) { return sizeof(int64_t) * (size_t)scan_words(n); }
cudaError_t exclusive_scan(const uint32_t* in, int64_t n, int64_t* scratch, uint32_t* out, cudaStream_t st,
                           int64_t* total) {
    return scan_counts<uint32_t, true>(in, n, scratch, out, total, st);
}
}  // namespace pgmpm

size_t pgmpm_hashgrid_s::layout(bool dense) {
    char* base = mem.as<char>();
    size_t at = 0;
    auto place = [&](auto*& p, size_t count) {
        p = base ? reinterpret_cast<std::remove_reference_t<decltype(p)>>(base + at) : nullptr;
        at += (sizeof(*p) * count + 255) & ~(size_t)255;
    };
    const size_t n = (size_t)stride(), cells = total;
    place(counts, cells);
    place(starts, cells);
    place(cell_ids, n);
    place(ka, n);
    place(va, n);
    place(kb, 2 * n);
    vb = kb ? kb + n : nullptr;
    place(scratch, (size_t)radix_sort_scratch_words((int64_t)n));
    place(stats, 3);
    place(scan, (size_t)scan_words((int64_t)std::max(n, cells)));
    place(result, 2);
    if (dense) {
        place(qcount, n);
        place(grid_rows, cells);
        place(grid_sum, cells);
        place(grid_first, cells + 1);
    }
    return at;
}

extern "C" {

int pgmpm_hashgrid_create(float cell_size, const float* domain_min, const float* domain_max, int64_t max_particles,
                          int32_t device, pgmpm_hashgrid* out) {
    if (!out || !domain_min || !domain_max) return fail(PGMPM_ERR_ARG, "hashgrid: null argument");
    *out = nullptr;
    if (!(cell_size > 0.f) || !std::isfinite(cell_size) || max_particles < 0 || max_particles > 0xFFFFFFFFll)
        return fail(PGMPM_ERR_ARG, "hashgrid: cell_size > 0 and 0 <= max_particles < 2^32 required");
    auto* g = new pgmpm_hashgrid_s();
    g->device = device;
    g->cell = cell_size;
    uint64_t total = 1;
    for (int a = 0; a < 3; ++a) {
        g->dmin[a] = domain_min[a];
        const float r = std::ceil((domain_max[a] - domain_min[a]) / cell_size);  // single precision, as the host class
        if (!(r >= 1.f) || !(r < 4294967296.f)) {
            delete g;
            return fail(PGMPM_ERR_ARG, "hashgrid: each axis needs 1 .. 2^32-1 cells");
        }
        g->res[a] = (uint32_t)r;
        total *= g->res[a];
        if (total > 0xFFFFFFFFull) {  // per factor: three of them overflow 64 bits
            delete g;
            return fail(PGMPM_ERR_ARG, "hashgrid: more than 2^32 - 1 cells");
        }
    }
    g->total = (uint32_t)total;
    g->key_bits = std::max(1, bits_for(total));
    g->max_particles = max_particles;
    DeviceGuard dg(device);
    // with the dense queries' tables (16 bytes per cell) where as many queries as
    // particles would use them
    const bool dense = (int64_t)total <= HG_DENSE_CELLS * max_particles && total < 0x80000000ull;
    cudaError_t e = g->mem.alloc(g->layout(dense));
    if (e == cudaSuccess) {
        g->layout(dense);
    } else if (dense) {
        cudaGetLastError();
        e = g->mem.alloc(g->layout(false));
        if (e == cudaSuccess) g->layout(false);
    }
    if (e != cudaSuccess) {
        cudaGetLastError();
        delete g;
        return fail(e == cudaErrorMemoryAllocation ? PGMPM_ERR_OOM : PGMPM_ERR_CUDA, "hashgrid: %s",
                    cudaGetErrorString(e));
    }
    *out = g;
    return PGMPM_OK;
}

int pgmpm_hashgrid_destroy(pgmpm_hashgrid g) {
    if (!g) return PGMPM_OK;
    DeviceGuard dg(g->device);
    delete g;
    return PGMPM_OK;
}

int pgmpm_hashgrid_build(pgmpm_hashgrid g, const float* positions, int64_t n, int32_t ptr_kind, void* stream) {
    if (!g || n < 0 || (n > 0 && !positions)) return fail(PGMPM_ERR_ARG, "hashgrid: bad arguments");
    if (n > g->max_particles) return fail(PGMPM_ERR_ARG, "hashgrid: more particles than max_particles");
    if (ptr_kind != PGMPM_PTR_HOST && ptr_kind != PGMPM_PTR_DEVICE) return fail(PGMPM_ERR_ARG, "bad ptr_kind");
    DeviceGuard dg(g->device);
    cudaStream_t st = ST(stream);
    int rc;
    const float* pos = staged(g->pos_stage, positions, 3 * n, ptr_kind, st, rc);
    if (rc) return rc;
    const HGDev G = dev_of(g);
    uint32_t *ids = g->cell_ids, *counts = g->counts;
    const uint32_t* sorted_index = nullptr;
    // per-cell counts (histogram of the cell ids), starts = their exclusive scan
    CK(cudaMemsetAsync(counts, 0, sizeof(uint32_t) * g->total, st));
    if (n > 0) {
        k_hg_cells<<<blocks_of(n, HG_T), HG_T, 0, st>>>(G, pos, n, ids, counts);
        CK(cudaGetLastError());
    }
    CK((scan_counts<uint32_t, false>(counts, g->total, g->scan, g->starts, nullptr, st)));
    // particles ordered by cell, by index within a cell (stable sort)
    if (n > 0) {
        int which = 0;
        CK(radix_sort_pairs(ids, nullptr, g->ka, g->va, g->kb, g->vb, g->scratch, n, g->key_bits, &which, st));
        sorted_index = which ? g->vb : g->va;
    }
    // keep the sorted indices where queries read them
    if (n > 0 && sorted_index != g->va)
        CK(cudaMemcpyAsync(g->va, sorted_index, sizeof(uint32_t) * n, cudaMemcpyDeviceToDevice, st));
    g->n = n;
    g->built = true;
    g->grid_ready = false;
    g->sum_src = -1;
    return PGMPM_OK;
}

int pgmpm_hashgrid_get_table(pgmpm_hashgrid g, uint32_t* counts, uint32_t* starts, uint32_t* particle_indices,
                             uint32_t* cell_ids, int32_t ptr_kind, void* stream) {
    if (!g || !g->built) return fail(PGMPM_ERR_STATE, "hashgrid: build first");
    if (ptr_kind != PGMPM_PTR_HOST && ptr_kind != PGMPM_PTR_DEVICE) return fail(PGMPM_ERR_ARG, "bad ptr_kind");
    DeviceGuard dg(g->device);
    cudaStream_t st = ST(stream);
    const cudaMemcpyKind k = ptr_kind == PGMPM_PTR_HOST ? cudaMemcpyDeviceToHost : cudaMemcpyDeviceToDevice;
    if (counts) CK(cudaMemcpyAsync(counts, g->counts, sizeof(uint32_t) * g->total, k, st));
    if (starts) CK(cudaMemcpyAsync(starts, g->starts, sizeof(uint32_t) * g->total, k, st));
    if (particle_indices && g->n) CK(cudaMemcpyAsync(particle_indices, g->va, sizeof(uint32_t) * g->n, k, st));
    if (cell_ids && g->n) CK(cudaMemcpyAsync(cell_ids, g->cell_ids, sizeof(uint32_t) * g->n, k, st));
    if (ptr_kind == PGMPM_PTR_HOST) CK(cudaStreamSynchronize(st));
    return PGMPM_OK;
}

int pgmpm_hashgrid_neighbors(pgmpm_hashgrid g, const float* queries, int64_t nq, float radius, int64_t* offsets,
                             uint32_t* indices, int64_t capacity, int64_t* total, int32_t ptr_kind, void* stream) {
    if (!g || !g->built) return fail(PGMPM_ERR_STATE, "hashgrid: build first");
    if (nq < 0 || (nq > 0 && !queries) || !offsets || !total || capacity < 0 || !(radius >= 0.f) ||
        !std::isfinite(radius))
        return fail(PGMPM_ERR_ARG, "hashgrid: bad query arguments");
    if (ptr_kind != PGMPM_PTR_HOST && ptr_kind != PGMPM_PTR_DEVICE) return fail(PGMPM_ERR_ARG, "bad ptr_kind");
    const float sr = std::ceil(radius / g->cell);  // single precision, as the host class
    // (2 src + 1)^3 cells per query must count in uint32
    if (!(sr < 512.f)) return fail(PGMPM_ERR_ARG, "hashgrid: radius spans more than 511 cells");
    const uint32_t src = (uint32_t)sr;
    DeviceGuard dg(g->device);
    cudaStream_t st = ST(stream);
    int rc;
    const float* q = staged(g->qstage, queries, 3 * nq, ptr_kind, st, rc);
    if (rc) return rc;
    const HGDev G = dev_of(g);
    const int64_t nb = scan_words(std::max<int64_t>(nq, 1));
    const size_t off_bytes = sizeof(int64_t) * (size_t)(nq + 1);
    int64_t* bsum = g->scan;
    uint32_t *qcount = g->qcount, *qcell = g->ka;
    if (nq > g->max_particles || !qcount) {
        CK(g->qlarge.ensure(sizeof(int64_t) * nb + 2 * sizeof(uint32_t) * std::max<int64_t>(nq, 1)));
        bsum = g->qlarge.as<int64_t>();
        qcount = reinterpret_cast<uint32_t*>(bsum + nb);
        qcell = qcount + nq;
    }
    if (ptr_kind == PGMPM_PTR_HOST) CK(g->off_stage.ensure(off_bytes));
    int64_t* doff = ptr_kind == PGMPM_PTR_HOST ? g->off_stage.as<int64_t>() : offsets;
    bool dense = false;
    const int64_t block = (int64_t)(2 * src + 1) * (2 * src + 1) * (2 * src + 1);
    if (g->grid_rows && (int64_t)g->total <= HG_DENSE_CELLS * nq && nq >= (HG_DENSE_WORK + block - 1) / block) {
        rc = dense_tables(g, G, src, st);
        if (rc < 0) return rc;
        dense = rc == 1;
    }
    auto fill = [&](uint32_t* dout, int64_t cap) {
        auto dfill = [&](auto kernel, int qw) {
            kernel<<<(int)std::min<int64_t>(blocks_of(nq, qw * (HG_T / 32)), 148 * 64), HG_T, 0, st>>>(
                G, q, nq, src, g->grid_first, g->grid_rows, g->index(), qcell, g->result + 1, g->index_capacity(), doff,
                cap, dout);
        };
        if (dense && src <= 1)  // 1 or 9 stretches per query
            src == 0 ? dfill(k_hg_dfill<32>, 32) : dfill(k_hg_dfill<3>, 3);
        else if (dense)
            dfill(k_hg_dfill<1>, 1);
        else
            k_hg_qfill<<<blocks_of(nq * HG_FG, HG_T), HG_T, 0, st>>>(G, q, nq, src, g->counts, g->starts, g->va, doff,
                                                                     dout);
    };
    int64_t tot = 0;
    bool filled = false;
    for (;; dense = false) {
        if (nq > 0) {
            if (dense)
                k_hg_dcount<<<blocks_of(nq, HG_T), HG_T, 0, st>>>(G, q, nq, src, g->grid_first, g->grid_sum, qcount,
                                                                  qcell);
            else
                k_hg_qcount<<<blocks_of(nq, HG_T), HG_T, 0, st>>>(G, q, nq, src, g->counts, qcount);
            CK((scan_counts<int64_t, true>(qcount, nq, bsum, doff, g->result, st)));
        } else {
            CK(cudaMemsetAsync(doff, 0, sizeof(int64_t), st));
            CK(cudaMemsetAsync(g->result, 0, sizeof(int64_t), st));
        }
        // into a device buffer the dense fill follows at once (it checks the
        // capacities itself); otherwise the host learns the total first
        filled = dense && indices && capacity > 0 && ptr_kind == PGMPM_PTR_DEVICE;
        if (filled) {
            fill(indices, capacity);
            CK(cudaGetLastError());
        }
        int64_t r[2] = {0, 0};
        CK(cudaMemcpyAsync(r, g->result, sizeof(int64_t) * (dense ? 2 : 1), cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
        tot = r[0];
        if (!dense || r[1] <= g->index_capacity()) break;
        // particles crowd in buckets that several cells share: hashed queries
        // now, a longer index for the next ones
        g->index_need = r[1];
        g->grid_ready = false;
    }
    *total = tot;
    if (ptr_kind == PGMPM_PTR_HOST) CK(cudaMemcpyAsync(offsets, doff, off_bytes, cudaMemcpyDeviceToHost, st));
    if (!filled && indices && tot <= capacity && tot > 0) {
        uint32_t* dout = indices;
        if (ptr_kind == PGMPM_PTR_HOST) {
            CK(g->qout_stage.ensure(sizeof(uint32_t) * tot));
            dout = g->qout_stage.as<uint32_t>();
        }
        fill(dout, tot);
        CK(cudaGetLastError());
        if (ptr_kind == PGMPM_PTR_HOST)
            CK(cudaMemcpyAsync(indices, dout, sizeof(uint32_t) * tot, cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
    } else if (ptr_kind == PGMPM_PTR_HOST) {
        CK(cudaStreamSynchronize(st));
    }
    return PGMPM_OK;
}

int pgmpm_hashgrid_stats(pgmpm_hashgrid g, pgmpm_hashgrid_info* out) {
    if (!g || !out) return fail(PGMPM_ERR_ARG, "hashgrid: null argument");
    DeviceGuard dg(g->device);
    unsigned long long h[3] = {0, 0, 0};  // before a build: no particles
    if (g->built) {
        CK(cudaMemset(g->stats, 0, sizeof(h)));
        k_hg_stats<<<std::min(blocks_of(g->total, HG_T), 148 * 8), HG_T>>>(g->counts, g->total, g->stats);
        CK(cudaGetLastError());
        CK(cudaMemcpy(h, g->stats, sizeof(h), cudaMemcpyDeviceToHost));
    }
    std::memset(out, 0, sizeof(*out));
    out->occupied_cells = (uint32_t)h[0];
    out->max_particles_per_cell = (uint32_t)h[1];
    out->average_particles_per_cell = (float)h[2] / (float)std::max<unsigned long long>(1, h[0]);
    out->load_factor = (float)h[0] / (float)g->total;
    // the host class's accounting: two words per cell and two per particle slot
    const double bytes = 2.0 * 4.0 * g->total + 2.0 * 4.0 * (double)g->max_particles;
    out->memory_usage_mb = (float)(bytes / (1024.0 * 1024.0));
    out->total_cells = g->total;
    for (int a = 0; a < 3; ++a) out->resolution[a] = g->res[a];
    return PGMPM_OK;
}

}  // extern "C"
