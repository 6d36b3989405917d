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
    DevBuf counts, starts;          // per cell
    DevBuf cell_ids;                // per particle: cell id (particle order)
    // sort buffers; between builds va keeps the sorted particle indices, ka and
    // vb are the dense queries' (dense_index, the queries' cells)
    DevBuf ka, va, kb, vb, scratch, pos_stage;
    DevBuf qcount, qstage, qout_stage, scan_tmp, stats;  // query scratch, kept between calls
    // dense queries (cells in grid order, x outer, z inner): z stretches and
    // block sums for the last half width and first[] of the cells' buckets (one
    // allocation), and the buckets themselves
    DevBuf grid_tables, grid_index;
    uint2* grid_rows() const { return grid_tables.as<uint2>(); }
    uint32_t* grid_sum() const { return reinterpret_cast<uint32_t*>(grid_rows() + total); }
    uint32_t* grid_first() const { return grid_sum() + total; }
    uint32_t* dense_index() const { return mult_max > 1 ? grid_index.as<uint32_t>() : vb.as<uint32_t>(); }
    uint32_t mult_max = 0;    // most cells that hash to one bucket (0: not counted yet)
    bool grid_ready = false;  // grid_first and grid_index hold the last build's
    int64_t sum_src = -1;     // grid_rows and grid_sum hold the last build's for this half width
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

// Fill pass, HG_FG lanes per query: they take the block's cells in the
// reference's order (linear index t = (dx (2s+1) + dy) (2s+1) + dz), HG_FG at
// a time, give each cell its place by a scan over the lanes and copy the
// cell's particles, so a query's list is written into one contiguous stretch
// by its lanes together.
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
// scan plus its carry.  A warp takes SCAN_ROWS rows of 32 counts, so that every
// access is a full line (2 M counts: sums 10 -> 3.9 us, apply 11.4 -> 7.7 us
// against one count per thread).
constexpr int SCAN_T = 1024;
constexpr int SCAN_ROWS = 4;
constexpr int SCAN_TILE = SCAN_T * SCAN_ROWS;  // counts per block
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
__global__ void __launch_bounds__(SCAN_T) k_scan_sums(const uint32_t* __restrict__ in, int64_t n,
                                                      int64_t* __restrict__ bsum) {
    __shared__ int64_t sh[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int64_t s = 0;
#pragma unroll
    for (int k = 0; k < SCAN_ROWS; ++k) {
        const int64_t i = (int64_t)blockIdx.x * SCAN_TILE + k * SCAN_T + threadIdx.x;
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
template <class OutT, bool TOTAL>
__global__ void __launch_bounds__(SCAN_T) k_scan_apply(const uint32_t* __restrict__ in, int64_t n,
                                                       const int64_t* __restrict__ bsum, OutT* __restrict__ out) {
    __shared__ int64_t sh[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t base = (int64_t)blockIdx.x * SCAN_TILE + warp * (32 * SCAN_ROWS) + lane;
    int64_t v[SCAN_ROWS], x[SCAN_ROWS], run = 0;
#pragma unroll
    for (int k = 0; k < SCAN_ROWS; ++k) v[k] = base + 32 * k < n ? in[base + 32 * k] : 0u;
#pragma unroll
    for (int k = 0; k < SCAN_ROWS; ++k) {  // inclusive over the warp's rows so far
        x[k] = run + warp_incl_scan(v[k], lane);
        run = __shfl_sync(0xFFFFFFFFu, x[k], 31);
    }
    if (lane == 0) sh[warp] = run;
    __syncthreads();
    if (warp == 0) sh[lane] = warp_incl_scan(sh[lane], lane);
    __syncthreads();
    const int64_t before = bsum[blockIdx.x] + (warp ? sh[warp - 1] : 0);
#pragma unroll
    for (int k = 0; k < SCAN_ROWS; ++k) {
        const int64_t i = base + 32 * k;
        if (i < n) out[i] = (OutT)(before + x[k] - v[k]);
        if (TOTAL && i == n - 1) out[n] = (OutT)(before + x[k]);
    }
}

// ------------------------------------------------------ dense query sets
// When the queries are at least 1/4 of the cells (HG_DENSE_CELLS), the index is first laid out
// again in grid order (x outer, z inner): every cell's bucket, one after the
// other, so that the 2s+1 cells of a query's block along z are one stretch of
// it and no query hashes anything:
//   k_hg_grid    (start, count) of every cell, scanned into the stretches
//   k_hg_expand  the buckets in grid order (buckets that several cells hash to
//                are repeated: at most mult_max times the particles)
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

__global__ void k_hg_mult(HGDev G, uint32_t* __restrict__ mult) {
    const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= G.total) return;
    const uint32_t z = c % G.res[2], xy = c / G.res[2], y = xy % G.res[1], x = xy / G.res[1];
    atomicAdd(&mult[hg_mod(hg_morton(x, y, z), G)], 1u);
}
__global__ void k_hg_max(const uint32_t* __restrict__ v, uint32_t n, uint32_t* __restrict__ out) {
    uint32_t m = 0;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) m = max(m, v[i]);
    m = __reduce_max_sync(0xFFFFFFFFu, m);
    if ((threadIdx.x & 31) == 0) atomicMax(out, m);
}
__global__ void k_hg_grid(HGDev G, const uint32_t* __restrict__ counts, const uint32_t* __restrict__ starts,
                          uint32_t* __restrict__ ccount, uint32_t* __restrict__ cstart) {
    const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= G.total) return;
    const uint32_t z = c % G.res[2], xy = c / G.res[2], y = xy % G.res[1], x = xy / G.res[1];
    const uint32_t id = hg_mod(hg_morton(x, y, z), G);
    ccount[c] = counts[id];
    cstart[c] = starts[id];
}
// first[c] .. first[c + 1]: cell c's bucket in grid order
__global__ void k_hg_expand(uint32_t total, const uint32_t* __restrict__ first, const uint32_t* __restrict__ cstart,
                            const uint32_t* __restrict__ sorted_index, uint32_t* __restrict__ out) {
    // warps copy their 32 cells' buckets together: one stretch of out
    const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t f = c < total ? first[c] : 0u, k = c < total ? first[c + 1] - f : 0u;
    const int lane = threadIdx.x & 31;
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
// Nothing is written when the lists (offsets[nq] entries) exceed capacity.
// QW: queries a warp takes together; their lists are one stretch of out, and
// (2 src + 1)^2 QW <= 32 stretches come from one read per lane.  QW = 1 also
// takes wider blocks, 32 stretches at a time.
template <int QW>
__global__ void __launch_bounds__(HG_T) k_hg_dfill(HGDev G, const float* __restrict__ q, int64_t nq, uint32_t src,
                                                   const uint32_t* __restrict__ first, const uint2* __restrict__ rows,
                                                   const uint32_t* __restrict__ index,
                                                   const uint32_t* __restrict__ qcell,
                                                   const int64_t* __restrict__ offsets, int64_t capacity,
                                                   uint32_t* __restrict__ out) {
    if (offsets[nq] > capacity) return;
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

// Cells per query up to which the dense tables pay: laying them out costs 30 ps
// per cell (2 M cells), and a hashed query of 27 cells 0.2 ns more than a dense
// one.
constexpr int64_t HG_DENSE_CELLS = 4;
constexpr uint32_t HG_DENSE_MULT = 8;  // most cells per bucket (grid_index is that many times the particles)

// The grid-order tables of the last build for blocks of half width src (kept
// until the next build).  1: ready; 0: too many cells share a bucket, or their
// memory is not to be had (the hashed queries need none); < 0: an error.
int dense_tables(pgmpm_hashgrid_s* g, const HGDev& G, uint32_t src, cudaStream_t st) {
    const size_t cells = g->total;
    const int nb = blocks_of((int64_t)cells, HG_T);
    const int64_t sb = ((int64_t)cells + SCAN_TILE - 1) / SCAN_TILE;
    auto have = [](cudaError_t e) {
        if (e != cudaSuccess) cudaGetLastError();  // clear the failed allocation
        return e == cudaSuccess;
    };
    if (!have(g->grid_tables.ensure((sizeof(uint2) + 2 * sizeof(uint32_t)) * cells + sizeof(uint32_t))) ||
        !have(g->scan_tmp.ensure(sizeof(int64_t) * sb)))
        return 0;
    uint32_t* sum = g->grid_sum();
    // a cube of 2^k cells an axis has no two cells in a bucket; otherwise count
    // once per grid, since it is a property of the resolution
    if (g->res[0] == g->res[1] && g->res[1] == g->res[2] && (g->res[0] & (g->res[0] - 1u)) == 0u) g->mult_max = 1;
    if (g->mult_max == 0) {
        CK(cudaMemsetAsync(sum, 0, sizeof(uint32_t) * cells, st));
        CK(cudaMemsetAsync(g->stats.p, 0, sizeof(uint32_t), st));
        k_hg_mult<<<nb, HG_T, 0, st>>>(G, sum);
        k_hg_max<<<std::min(nb, 148 * 8), HG_T, 0, st>>>(sum, g->total, g->stats.as<uint32_t>());
        CK(cudaGetLastError());
        CK(cudaMemcpyAsync(&g->mult_max, g->stats.p, sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
    }
    // with a cell per bucket the copy is as long as the particles, and takes a
    // buffer of the build's sort (the first query of 2 M on a new grid 1771 -> 1250 us)
    if (g->mult_max > HG_DENSE_MULT || g->n * g->mult_max > 0xFFFFFFFFll ||
        (g->mult_max > 1 && !have(g->grid_index.ensure(sizeof(uint32_t) * std::max<size_t>((size_t)g->n * g->mult_max, 1)))))
        return 0;
    uint32_t* first = g->grid_first();
    if (!g->grid_ready) {
        uint32_t* cstart = reinterpret_cast<uint32_t*>(g->grid_rows());  // until k_hg_rows writes it
        int64_t* bsum = g->scan_tmp.as<int64_t>();
        k_hg_grid<<<nb, HG_T, 0, st>>>(G, g->counts.as<uint32_t>(), g->starts.as<uint32_t>(), sum, cstart);
        CK(exclusive_scan(sum, (int64_t)cells, bsum, first, st));
        k_hg_expand<<<nb, HG_T, 0, st>>>(g->total, first, cstart, g->va.as<uint32_t>(), g->dense_index());
    }
    if (!g->grid_ready || g->sum_src != (int64_t)src) {
        k_hg_rows<<<nb, HG_T, 0, st>>>(G, src, first, g->grid_rows());
        k_hg_blocks<<<nb, HG_T, 0, st>>>(G, src, g->grid_rows(), sum);
    }
    CK(cudaGetLastError());
    g->grid_ready = true;
    g->sum_src = src;
    return 1;
}

}  // namespace

namespace pgmpm {
size_t exclusive_scan_bytes(int64_t n) { return sizeof(int64_t) * (size_t)((n + SCAN_TILE - 1) / SCAN_TILE); }
cudaError_t exclusive_scan(const uint32_t* in, int64_t n, int64_t* scratch, uint32_t* out, cudaStream_t st) {
    const int64_t nb = (n + SCAN_TILE - 1) / SCAN_TILE;
    k_scan_sums<<<(int)nb, SCAN_T, 0, st>>>(in, n, scratch);
    k_scan_carry<<<1, SCAN_T, 0, st>>>(scratch, nb);
    k_scan_apply<uint32_t, true><<<(int)nb, SCAN_T, 0, st>>>(in, n, scratch, out);
    return cudaGetLastError();
}
}  // namespace pgmpm

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
    const size_t n = (size_t)std::max<int64_t>(max_particles, 1);
    cudaError_t e = g->counts.alloc(sizeof(uint32_t) * total);
    if (e == cudaSuccess) e = g->starts.alloc(sizeof(uint32_t) * total);
    if (e == cudaSuccess) e = g->cell_ids.alloc(sizeof(uint32_t) * n);
    if (e == cudaSuccess) e = g->ka.alloc(sizeof(uint32_t) * n);
    if (e == cudaSuccess) e = g->va.alloc(sizeof(uint32_t) * n);
    if (e == cudaSuccess) e = g->kb.alloc(sizeof(uint32_t) * n);
    if (e == cudaSuccess) e = g->vb.alloc(sizeof(uint32_t) * n);
    if (e == cudaSuccess) e = g->scratch.alloc(sizeof(uint32_t) * radix_sort_scratch_words((int64_t)n));
    if (e == cudaSuccess) e = g->stats.alloc(sizeof(unsigned long long) * 3);
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
    uint32_t* ids = g->cell_ids.as<uint32_t>();
    uint32_t* counts = g->counts.as<uint32_t>();
    const uint32_t* sorted_index = nullptr;
    // per-cell counts (histogram of the cell ids), starts = their exclusive scan
    CK(cudaMemsetAsync(counts, 0, sizeof(uint32_t) * g->total, st));
    if (n > 0) {
        k_hg_cells<<<blocks_of(n, HG_T), HG_T, 0, st>>>(G, pos, n, ids, counts);
        CK(cudaGetLastError());
    }
    const int64_t nb = ((int64_t)g->total + SCAN_TILE - 1) / SCAN_TILE;
    CK(g->scan_tmp.ensure(sizeof(int64_t) * nb));
    int64_t* bsum = g->scan_tmp.as<int64_t>();
    k_scan_sums<<<(int)nb, SCAN_T, 0, st>>>(counts, g->total, bsum);
    k_scan_carry<<<1, SCAN_T, 0, st>>>(bsum, nb);
    k_scan_apply<uint32_t, false><<<(int)nb, SCAN_T, 0, st>>>(counts, g->total, bsum, g->starts.as<uint32_t>());
    CK(cudaGetLastError());
    // particles ordered by cell, by index within a cell (stable sort)
    if (n > 0) {
        int which = 0;
        CK(radix_sort_pairs(ids, nullptr, g->ka.as<uint32_t>(), g->va.as<uint32_t>(), g->kb.as<uint32_t>(),
                            g->vb.as<uint32_t>(), g->scratch.as<uint32_t>(), n, g->key_bits, &which, st));
        sorted_index = which ? g->vb.as<uint32_t>() : g->va.as<uint32_t>();
    }
    // keep the sorted indices where queries read them
    if (n > 0 && sorted_index != g->va.as<uint32_t>())
        CK(cudaMemcpyAsync(g->va.p, sorted_index, sizeof(uint32_t) * n, cudaMemcpyDeviceToDevice, st));
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
    if (counts) CK(cudaMemcpyAsync(counts, g->counts.p, sizeof(uint32_t) * g->total, k, st));
    if (starts) CK(cudaMemcpyAsync(starts, g->starts.p, sizeof(uint32_t) * g->total, k, st));
    if (particle_indices && g->n) CK(cudaMemcpyAsync(particle_indices, g->va.p, sizeof(uint32_t) * g->n, k, st));
    if (cell_ids && g->n) CK(cudaMemcpyAsync(cell_ids, g->cell_ids.p, sizeof(uint32_t) * g->n, k, st));
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
    // counts, then the queries' cells, unless those fit a buffer of the build's sort
    const bool reuse = nq <= g->max_particles;
    CK(g->qcount.ensure((reuse ? 1 : 2) * sizeof(uint32_t) * std::max<int64_t>(nq, 1)));
    const int64_t nb = std::max<int64_t>(1, (nq + SCAN_TILE - 1) / SCAN_TILE);
    const size_t off_bytes = sizeof(int64_t) * (size_t)(nq + 1);
    uint32_t *qcount = g->qcount.as<uint32_t>(), *qcell = reuse ? g->ka.as<uint32_t>() : qcount + nq;
    bool dense = false;
    if (nq > 0 && (int64_t)g->total <= HG_DENSE_CELLS * nq && g->total < 0x80000000u) {
        rc = dense_tables(g, G, src, st);
        if (rc < 0) return rc;
        dense = rc == 1;
    }
    // scan_tmp: block sums, then the offsets when the caller's are on the host
    CK(g->scan_tmp.ensure(sizeof(int64_t) * nb + (ptr_kind == PGMPM_PTR_HOST ? off_bytes : 0)));
    int64_t* bsum = g->scan_tmp.as<int64_t>();
    int64_t* doff = ptr_kind == PGMPM_PTR_HOST ? bsum + nb : offsets;
    const uint32_t* first = dense ? g->grid_first() : nullptr;
    if (nq > 0) {
        if (dense)
            k_hg_dcount<<<blocks_of(nq, HG_T), HG_T, 0, st>>>(G, q, nq, src, first, g->grid_sum(), qcount,
                                                              qcell);
        else
            k_hg_qcount<<<blocks_of(nq, HG_T), HG_T, 0, st>>>(G, q, nq, src, g->counts.as<uint32_t>(), qcount);
        k_scan_sums<<<(int)nb, SCAN_T, 0, st>>>(qcount, nq, bsum);
        k_scan_carry<<<1, SCAN_T, 0, st>>>(bsum, nb);
        k_scan_apply<int64_t, true><<<(int)nb, SCAN_T, 0, st>>>(qcount, nq, bsum, doff);
        CK(cudaGetLastError());
    } else {
        CK(cudaMemsetAsync(doff, 0, sizeof(int64_t), st));
    }
    auto fill = [&](uint32_t* dout, int64_t cap) {
        auto dfill = [&](auto kernel, int qw) {
            kernel<<<(int)std::min<int64_t>(blocks_of(nq, qw * (HG_T / 32)), 148 * 64), HG_T, 0, st>>>(
                G, q, nq, src, first, g->grid_rows(), g->dense_index(), qcell,
                doff, cap, dout);
        };
        if (dense && src <= 1)  // 1 or 9 stretches per query
            src == 0 ? dfill(k_hg_dfill<32>, 32) : dfill(k_hg_dfill<3>, 3);
        else if (dense)
            dfill(k_hg_dfill<1>, 1);
        else
            k_hg_qfill<<<blocks_of(nq * HG_FG, HG_T), HG_T, 0, st>>>(G, q, nq, src, g->counts.as<uint32_t>(),
                                                                     g->starts.as<uint32_t>(), g->va.as<uint32_t>(),
                                                                     doff, dout);
    };
    // into a device buffer the dense fill follows at once (it checks the
    // capacity itself); otherwise the host learns the total first
    const bool early = dense && indices && capacity > 0 && ptr_kind == PGMPM_PTR_DEVICE;
    if (early) {
        fill(indices, capacity);
        CK(cudaGetLastError());
    }
    int64_t tot = 0;
    CK(cudaMemcpyAsync(&tot, doff + nq, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    *total = tot;
    if (ptr_kind == PGMPM_PTR_HOST) CK(cudaMemcpyAsync(offsets, doff, off_bytes, cudaMemcpyDeviceToHost, st));
    if (!early && indices && tot <= capacity && tot > 0) {
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
        CK(cudaMemset(g->stats.p, 0, sizeof(h)));
        k_hg_stats<<<std::min(blocks_of(g->total, HG_T), 148 * 8), HG_T>>>(g->counts.as<uint32_t>(), g->total,
                                                                          g->stats.as<unsigned long long>());
        CK(cudaGetLastError());
        CK(cudaMemcpy(h, g->stats.p, sizeof(h), cudaMemcpyDeviceToHost));
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
