// pgmpm_sort.cu -- stable LSD radix sort of (u32 key, u32 value) pairs.
//
// Each pass sorts by one digit of `bits` (<= 8) bits with three kernels:
//   rs_hist     per-block digit histogram of a 2048-key tile (warp-aggregated
//               shared atomics), written digit-major hist[d][block]
//   rs_scan     one block per digit: exclusive scan of its row over blocks,
//               row totals to totals[d]
//   rs_scatter  block-local stable rank (per-warp ranking with match_any,
//               warp prefix per digit), keys staged in shared memory in
//               block-sorted order, then written out so that consecutive
//               threads store consecutive positions of a digit run.
// Stability: inside a block, warps own contiguous 256-key ranges processed
// in order, lanes in order; across blocks, the digit-major exclusive scan
// orders blocks.  The result is therefore identical to a stable CPU sort.
// Scratch: hist (digits x blocks u32), totals (256 u32), and ping-pong
// (key, value) buffers of n pairs, provided by the caller.
#include <algorithm>

#include "pgmpm_internal.h"

namespace pgmpm {

namespace {
constexpr int RS_THREADS = 256;
constexpr int RS_WARPS = RS_THREADS / 32;
constexpr int RS_ITEMS = 8;  // keys per thread per tile
constexpr int RS_TILE = RS_THREADS * RS_ITEMS;
constexpr int RS_MAXD = 256;
static_assert(RS_TILE == RADIX_TILE && RS_MAXD == RADIX_MAX_DIGITS, "scratch sizing must match the kernels");

__global__ void __launch_bounds__(RS_THREADS) rs_hist(const uint32_t* keys, int64_t n, int shift, int bits,
                                                      uint32_t* hist, int nblocks) {
    step_wait();
    // warp-private histograms with native integer shared atomics, summed at the end
    __shared__ uint32_t cnt[RS_WARPS][RS_MAXD];
    const int nd = 1 << bits;
    const uint32_t mask = (uint32_t)nd - 1u;
    for (int d = threadIdx.x; d < RS_WARPS * RS_MAXD; d += RS_THREADS) (&cnt[0][0])[d] = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t base = (int64_t)blockIdx.x * RS_TILE + warp * (32 * RS_ITEMS);
    uint32_t k[RS_ITEMS];
#pragma unroll
    for (int r = 0; r < RS_ITEMS; ++r) {
        const int64_t i = base + r * 32 + lane;
        k[r] = i < n ? keys[i] : 0u;
    }
#pragma unroll
    for (int r = 0; r < RS_ITEMS; ++r) {
        const int64_t i = base + r * 32 + lane;
        if (i < n) atomicAdd(&cnt[warp][(k[r] >> shift) & mask], 1u);
    }
    __syncthreads();
    for (int d = threadIdx.x; d < nd; d += RS_THREADS) {
        uint32_t s = 0;
#pragma unroll
        for (int w = 0; w < RS_WARPS; ++w) s += cnt[w][d];
        hist[(int64_t)d * nblocks + blockIdx.x] = s;
    }
}

// Lanes of the warp holding the same digit as this lane (bits <= 8), built
// from one ballot per digit bit; only lanes with `ok` participate.
__device__ __forceinline__ uint32_t digit_peers(uint32_t d, int bits, bool ok) {
    uint32_t peers = __ballot_sync(0xFFFFFFFFu, ok);
    if (!ok) peers = ~peers;
    for (int b = 0; b < bits; ++b) {
        const bool bit = (d >> b) & 1u;
        const uint32_t bal = __ballot_sync(0xFFFFFFFFu, bit);
        peers &= bit ? bal : ~bal;
    }
    return peers;
}

// Block-wide exclusive scan of one value per thread (blockDim.x <= 1024).
__device__ __forceinline__ uint32_t block_excl_scan(uint32_t v, uint32_t* sh, uint32_t& total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) sh[warp] = x;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = lane < nw ? sh[lane] : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t y = __shfl_up_sync(0xFFFFFFFFu, w, o);
            if (lane >= o) w += y;
        }
        sh[lane] = w;  // inclusive warp totals
    }
    __syncthreads();
    const uint32_t before = warp > 0 ? sh[warp - 1] : 0u;
    total = sh[nw - 1];
    __syncthreads();
    return before + x - v;
}

__global__ void __launch_bounds__(1024) rs_scan(uint32_t* hist, int nblocks, uint32_t* totals) {
    step_wait();
    __shared__ uint32_t sh[32];
    uint32_t* row = hist + (int64_t)blockIdx.x * nblocks;
    uint32_t carry = 0;
    for (int b0 = 0; b0 < nblocks; b0 += blockDim.x) {
        const int b = b0 + threadIdx.x;
        const uint32_t v = b < nblocks ? row[b] : 0u;
        uint32_t tot;
        const uint32_t ex = block_excl_scan(v, sh, tot);
        if (b < nblocks) row[b] = carry + ex;
        carry += tot;
    }
    if (threadIdx.x == 0) totals[blockIdx.x] = carry;
}

__global__ void __launch_bounds__(RS_THREADS) rs_scatter(const uint32_t* kin, const uint32_t* vin, uint32_t* kout,
                                                         uint32_t* vout, int64_t n, int shift, int bits,
                                                         const uint32_t* hist, int nblocks, const uint32_t* totals) {
    step_wait();
    __shared__ uint32_t wcnt[RS_WARPS][RS_MAXD];
    __shared__ uint32_t boff[RS_MAXD];   // block-local exclusive digit offsets
    __shared__ uint32_t goff[RS_MAXD];   // global position of this block's first key of digit d
    __shared__ uint32_t skey[RS_TILE];
    __shared__ uint32_t sval[RS_TILE];
    __shared__ uint32_t sh[32];
    const int nd = 1 << bits;
    const uint32_t mask = (uint32_t)nd - 1u;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t tile0 = (int64_t)blockIdx.x * RS_TILE;
    const int64_t base = tile0 + warp * (32 * RS_ITEMS);
    // All reads first: among the ranking's barriers each of the 8 waited alone
    // (a pass over 4,096 keys 7.3 -> 5.2 us, over 2 M 19 -> 16 us).  Its ballots
    // in a loop over the digit's bits: unrolled 4.9 and 16.9 us, __match_any 4.8
    // and 21 us.
    uint32_t k[RS_ITEMS], v[RS_ITEMS], rk[RS_ITEMS];
#pragma unroll
    for (int r = 0; r < RS_ITEMS; ++r) {
        const int64_t i = base + r * 32 + lane;
        k[r] = i < n ? kin[i] : 0xFFFFFFFFu;
        v[r] = i < n ? (vin ? vin[i] : (uint32_t)i) : 0u;
    }
    for (int d = threadIdx.x; d < RS_WARPS * RS_MAXD; d += RS_THREADS) (&wcnt[0][0])[d] = 0;
    // global digit prefix (exclusive scan of totals) + this block's row offset
    {
        const uint32_t t = threadIdx.x < nd ? totals[threadIdx.x] : 0u;
        uint32_t tot;
        const uint32_t ex = block_excl_scan(t, sh, tot);
        if (threadIdx.x < nd) goff[threadIdx.x] = ex + hist[(int64_t)threadIdx.x * nblocks + blockIdx.x];
    }
    __syncthreads();
    const uint32_t lt = (1u << lane) - 1u;
#pragma unroll
    for (int r = 0; r < RS_ITEMS; ++r) {
        const int64_t i = base + r * 32 + lane;
        const bool ok = i < n;
        const uint32_t d = ok ? ((k[r] >> shift) & mask) : 0u;
        const uint32_t peers = digit_peers(d, bits, ok);
        uint32_t c = 0u;
        if (ok) c = wcnt[warp][d];
        rk[r] = c + (uint32_t)__popc(peers & lt);
        __syncwarp();
        if (ok && lane == __ffs(peers) - 1) wcnt[warp][d] = c + (uint32_t)__popc(peers);
        __syncwarp();
    }
    __syncthreads();
    // per digit: exclusive prefix over warps, and block total
    uint32_t mytot = 0u;
    if (threadIdx.x < nd) {
        uint32_t run = 0u;
#pragma unroll
        for (int w = 0; w < RS_WARPS; ++w) {
            const uint32_t c = wcnt[w][threadIdx.x];
            wcnt[w][threadIdx.x] = run;
            run += c;
        }
        mytot = run;
    }
    {
        uint32_t tot;
        const uint32_t ex = block_excl_scan(mytot, sh, tot);
        if (threadIdx.x < nd) boff[threadIdx.x] = ex;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < RS_ITEMS; ++r) {
        const int64_t i = base + r * 32 + lane;
        if (i < n) {
            const uint32_t d = (k[r] >> shift) & mask;
            const uint32_t lp = boff[d] + wcnt[warp][d] + rk[r];
            if (lp < (uint32_t)RS_TILE) {
                skey[lp] = k[r];
                sval[lp] = v[r];
            }
        }
    }
    __syncthreads();
    const int cnt = (int)min((int64_t)RS_TILE, n - tile0);
    for (int j = threadIdx.x; j < cnt; j += RS_THREADS) {
        const uint32_t kk = skey[j];
        const uint32_t d = (kk >> shift) & mask;
        const uint32_t pos = goff[d] + (uint32_t)j - boff[d];
        if ((int64_t)pos < n) {
            kout[pos] = kk;
            vout[pos] = sval[j];
        }
    }
}

// --------------------------------------------------- per-step bin sort
// The MPM step groups particles by cell with a counting sort over the cells
// (key = cell tile << 6 | cell in tile) instead of a full radix sort:
//   bs_count     particles per cell and per cell tile, and each particle's
//                slot in its cell.  Lanes holding equal keys
//                in a run (the physical order stays close to cell order)
//                share one atomic: the run's first lane adds the run length.
//                Launched for the first step of a call only: the G2P of a
//                step that another one follows counts the keys it writes.
//   bs_groups    on grids of more than BS_DIRECT_TILES cell tiles: sums of the
//                tile counts over groups of BS_GROUP tiles.
//   bs_tiles     (a) one block per 8 or 64 cell tiles: sums the counts before
//                its range, and one warp per occupied tile scans its 64 cell
//                counts -> every cell's range, clearing the cell
//                counters, and lists the tile with its rank in its size
//                class; (b) one thread per node tile: active iff one of the 8
//                cell tiles around it is occupied.
//   bs_scatter   particle -> cell begin + slot; the occupied tiles' places in
//                the largest-first list P2G takes work from (the last tiles a
//                persistent P2G block picks up are then small ones, which
//                shortens the kernel's tail); clears the tile counters and
//                publishes the step's counter words.
// The counters are left zero for the next step by their readers, so a step
// costs O(N + occupied cells + tiles) with no clearing pass.  Keys come out
// sorted; particles that share a cell in atomic-arrival order, which the
// step does not rely on.
//
// Small scenes are bound by the launches (each kernel is a chain of a few
// dependent L2 reads, 3-5 us), large ones by the passes over the particles:
// counting inside G2P, where the keys are in registers, and scanning tiles
// and cells in one kernel took the sort from four kernels to two per step: 50
// steps of 32,768 particles 2148 -> 1725 us, 20 steps of 2 M particles (which
// keep the counting pass) 5464 -> 5308 us.
constexpr int BS_T = 256;
constexpr int BS_ITEMS = 8;                 // keys per thread in bs_count / bs_scatter
constexpr int BS_TILE = BS_T * BS_ITEMS;    // keys per block
constexpr int BS_REC_ITEMS = 1;             // particles per thread of bs_scatter when it moves their records
// cell tiles per warp of bs_tiles: a warp takes its occupied tiles in turn
// (~1 us each: a sparse grid's claims are chains of L2 reads), so few per warp
// are better until the blocks' reads of the counts before them (tiles^2 / 2
// words over all blocks) outgrow that
constexpr int BT_FEW = 1, BT_MANY = 8;
constexpr int64_t BT_FEW_TILES = 8192;      // most cell tiles for BT_FEW
constexpr int64_t BS_DIRECT_TILES = 65536;  // most cell tiles whose counts bs_tiles sums without bs_groups
constexpr int BS_GROUP = 1024;              // cell tiles per group of bs_groups

// Run structure of `bin` over a warp: first lane of this lane's run and one
// past its last lane.  A run is a maximal stretch of consecutive lanes with
// the same bin and the same ok.
__device__ __forceinline__ void bs_run(uint32_t bin, bool ok, int lane, int& start, int& end) {
    const uint32_t prev = __shfl_up_sync(0xFFFFFFFFu, bin, 1);
    const uint32_t okp = __shfl_up_sync(0xFFFFFFFFu, (uint32_t)ok, 1);
    const bool head = lane == 0 || bin != prev || (uint32_t)ok != okp;
    const uint32_t heads = __ballot_sync(0xFFFFFFFFu, head);
    const uint32_t upto = lane == 31 ? 0xFFFFFFFFu : ((2u << lane) - 1u);  // lanes <= this one
    start = 31 - __clz(heads & upto);
    const uint32_t after = heads & ~upto;
    end = after ? __ffs(after) - 1 : 32;
}

__global__ void __launch_bounds__(BS_T) bs_count(const uint32_t* keys, int64_t n, SortCounts c, uint32_t* counters) {
    step_wait();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // a new step stamp (sparse grids mark active node tiles with it)
    if (blockIdx.x == 0 && threadIdx.x == 0) counters[CNT_STAMP] += 1u;
    const int64_t base = (int64_t)blockIdx.x * BS_TILE + warp * (32 * BS_ITEMS);
    uint32_t k[BS_ITEMS], cb[BS_ITEMS];
    int st[BS_ITEMS];
    bool bad = false;
#pragma unroll
    for (int r = 0; r < BS_ITEMS; ++r) {
        const int64_t i = base + r * 32 + lane;
        k[r] = i < n ? keys[i] : 0u;
        if (i < n && k[r] >= c.ncells) {  // out-of-range key: overflow bin after the last cell
            bad = true;
            k[r] = c.ncells;
        }
    }
#pragma unroll
    for (int r = 0; r < BS_ITEMS; ++r) {
        const bool ok = base + r * 32 + lane < n;
        int e, ts, te;
        bs_run(k[r], ok, lane, st[r], e);
        bs_run(k[r] >> 6, ok, lane, ts, te);
        cb[r] = 0u;
        if (ok && lane == st[r]) cb[r] = atomicAdd(&c.ccount[k[r]], (uint32_t)(e - st[r]));
        if (ok && lane == ts) atomicAdd(&c.tcount[k[r] >> 6], (uint32_t)(te - ts));
    }
#pragma unroll
    for (int r = 0; r < BS_ITEMS; ++r) {
        const int64_t i = base + r * 32 + lane;
        const uint32_t b = __shfl_sync(0xFFFFFFFFu, cb[r], st[r]);
        if (i < n) c.slot[i] = b + (uint32_t)(lane - st[r]);
    }
    if (bad) atomicOr(&counters[CNT_FLAGS], FLAG_TILE_RANGE);
}

// Warp-aggregated append of `item` (lanes with want) to list / counter;
// returns the slot written (meaningful where want).
__device__ __forceinline__ uint32_t bs_append(uint32_t* list, uint32_t* counter, bool want, uint32_t item,
                                              int lane) {
    const uint32_t m = __ballot_sync(0xFFFFFFFFu, want);
    if (!m) return 0u;
    const int leader = __ffs(m) - 1;
    uint32_t b = 0;
    if (lane == leader) b = atomicAdd(counter, (uint32_t)__popc(m));
    b = __shfl_sync(0xFFFFFFFFu, b, leader);
    const uint32_t slot = b + __popc(m & ((1u << lane) - 1u));
    if (want && list) list[slot] = item;
    return slot;
}

// Size class of an occupied tile, 0 = largest (>= 1024 particles) ...
// CNT_BUCKETS - 1 = smallest (< 16).
__device__ __forceinline__ int bs_class(uint32_t count) {
    const int lg = 31 - __clz(count);  // count >= 1
    return min(CNT_BUCKETS - 1, max(0, 10 - lg));
}

// tcount holds a multiple of 4 words past the tiles' and the overflow bin's
// (zero), so a group of BS_GROUP or a run of 4 may be read whole
__global__ void __launch_bounds__(BS_T) bs_groups(const uint32_t* tcount, int64_t n, uint32_t* gsum) {
    step_wait();
    static_assert(BS_GROUP == 4 * BS_T, "one 16-byte load per thread");
    __shared__ uint32_t s_sum[BS_T / 32];
    const int64_t i = (int64_t)blockIdx.x * BS_GROUP + 4 * threadIdx.x;
    const uint4 c = i < n ? *reinterpret_cast<const uint4*>(tcount + i) : make_uint4(0u, 0u, 0u, 0u);
    const uint32_t w = __reduce_add_sync(0xFFFFFFFFu, c.x + c.y + c.z + c.w);
    if ((threadIdx.x & 31) == 0) s_sum[threadIdx.x >> 5] = w;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t t = 0u;
#pragma unroll
        for (int k = 0; k < BS_T / 32; ++k) t += s_sum[k];
        gsum[blockIdx.x] = t;
    }
}

// Blocks [0, cell_blocks): (a), the rest: (b).  See the overview above.
// gsum: the groups' sums, or null where the tile counts are summed directly.
template <int BT_PER_WARP>
__global__ void __launch_bounds__(BS_T) bs_tiles(View V, SortCounts c, const uint32_t* gsum, uint2* cell_range,
                                                 uint4* tile_info, int cell_blocks) {
    step_wait();
    constexpr int BT_TILES = BT_PER_WARP * (BS_T / 32);
    static_assert(BT_TILES <= 64 && BT_TILES % 4 == 0, "two tiles per lane in the scan, 16-byte reads of the counts");
    __shared__ uint32_t s_cnt[BT_TILES], s_slot[BT_TILES], s_rank[BT_TILES], s_sum[BS_T / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if ((int)blockIdx.x < cell_blocks) {
        const int64_t t0 = (int64_t)blockIdx.x * BT_TILES;
        uint32_t cnt = 0u;
        if (threadIdx.x < BT_TILES) {
            const int64_t t = t0 + threadIdx.x;
            cnt = t < (int64_t)V.total_ct ? c.tcount[t] : 0u;
            s_cnt[threadIdx.x] = cnt;
        }
        if (blockIdx.x == 0 && threadIdx.x == 0) V.sort_work[SW_VALID] = (uint32_t)V.N - c.tcount[V.total_ct];
        if (!__syncthreads_or(cnt > 0u)) return;
        // this warp's cell counts, in flight while the offsets are summed
        uint2 cc[BT_PER_WARP];
#pragma unroll
        for (int j = 0; j < BT_PER_WARP; ++j) {
            const int i = warp * BT_PER_WARP + j;
            cc[j] = s_cnt[i] ? reinterpret_cast<const uint2*>(c.ccount + (size_t)(t0 + i) * 64)[lane]
                             : make_uint2(0u, 0u);
        }
        // particles in the tiles before this block's: whole groups, then tiles
        uint32_t part = 0u;
        int64_t first = 0;
        if (gsum) {
            const int64_t g = t0 / BS_GROUP;
            for (int64_t i = threadIdx.x; i < g; i += BS_T) part += gsum[i];
            first = g * BS_GROUP;
        }
#pragma unroll 8
        for (int64_t i = first + 4 * threadIdx.x; i < t0; i += 4 * BS_T) {
            const uint4 w = *reinterpret_cast<const uint4*>(c.tcount + i);  // t0 is a multiple of 4
            part += w.x + w.y + w.z + w.w;
        }
        part = __reduce_add_sync(0xFFFFFFFFu, part);
        if (lane == 0) s_sum[warp] = part;
        if (threadIdx.x < (BT_TILES < 32 ? 32 : BT_TILES)) {  // whole warps
            const bool occ = cnt > 0u;
            const uint32_t lslot = bs_append(nullptr, &V.sort_work[SW_CTILES], occ, 0u, lane);
            // rank inside the tile's size class (lanes of one class share an atomic)
            const uint32_t cls = occ ? (uint32_t)bs_class(cnt) : (uint32_t)(CNT_BUCKETS + lane);
            const uint32_t peers = __match_any_sync(0xFFFFFFFFu, cls);
            const int leader = __ffs(peers) - 1;
            uint32_t b = 0;
            if (occ && lane == leader) b = atomicAdd(&V.sort_work[SW_BUCKET + cls], (uint32_t)__popc(peers));
            b = __shfl_sync(0xFFFFFFFFu, b, leader);
            if (occ) {
                s_slot[threadIdx.x] = lslot;
                s_rank[threadIdx.x] = (cls << 28) | (b + (uint32_t)__popc(peers & ((1u << lane) - 1u)));
            }
        }
        __syncthreads();
        uint32_t base = 0u;
#pragma unroll
        for (int w = 0; w < BS_T / 32; ++w) base += s_sum[w];
        // exclusive scan of the block's tile counts, tiles 2 lane and 2 lane + 1 per lane
        const uint32_t ca = 2 * lane < BT_TILES ? s_cnt[2 * lane] : 0u;
        const uint32_t cb = 2 * lane < BT_TILES ? s_cnt[2 * lane + 1] : 0u;
        uint32_t tx = ca + cb;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, tx, o);
            if (lane >= o) tx += y;
        }
        const uint32_t te = base + tx - ca - cb;  // first position of tile 2 lane
#pragma unroll
        for (int j = 0; j < BT_PER_WARP; ++j) {
            const int i = warp * BT_PER_WARP + j;
            const uint32_t tcnt = s_cnt[i];
            const uint32_t tb = __shfl_sync(0xFFFFFFFFu, (i & 1) ? te + ca : te, i >> 1);
            if (tcnt == 0u) continue;
            const uint32_t t = (uint32_t)t0 + (uint32_t)i;
            uint32_t x = cc[j].x + cc[j].y;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
                if (lane >= o) x += y;
            }
            const uint32_t e = tb + x - cc[j].x - cc[j].y;  // first position of cell 2 lane
            reinterpret_cast<uint4*>(cell_range + (size_t)t * 64)[lane] =
                make_uint4(e, e + cc[j].x, e + cc[j].x, e + cc[j].x + cc[j].y);
            reinterpret_cast<uint2*>(c.ccount + (size_t)t * 64)[lane] = make_uint2(0u, 0u);  // clear for the next step
            if (lane == 0) tile_info[s_slot[i]] = make_uint4(t, tb, tb + tcnt, s_rank[i]);
            if (V.sp.cap) {
                // sparse grid: lanes 0..7 find (or claim) the slots of the 8
                // node tiles the cell tile's stencils reach, list them for the
                // tile, and mark them active for this step (the first marker
                // appends the tile to the active list)
                uint32_t nslot = SP_NONE;
                uint32_t f = 0;
                if (lane < 8) {
                    int sx, sy, sz;
                    sp_decode(V.sp.code[t], sx, sy, sz);
                    nslot = sp_find_or_insert(V.sp, sp_code(sx + (lane & 1), sy + ((lane >> 1) & 1), sz + (lane >> 2)),
                                              f);
                    reinterpret_cast<uint32_t*>(V.sp.nbr + 2 * (size_t)t)[lane] = nslot == SP_NONE ? 0u : nslot;
                }
                if (f) atomicOr(&V.counters[CNT_FLAGS], f);
                const uint32_t stamp = V.counters[CNT_STAMP];
                // node tile nslot lies at offset `lane` of this tile's box (one
                // writer per (node tile, offset): t = nslot - offset)
                if (lane < 8 && nslot != SP_NONE) V.sp.rev[8 * (size_t)nslot + lane] = make_uint2(t, stamp);
                const bool fresh = lane < 8 && nslot != SP_NONE && atomicExch(&V.tile_flags[nslot], stamp) != stamp;
                bs_append(V.tile_list, &V.sort_work[SW_TILES], fresh, nslot, lane);
            }
        }
        return;
    }
    const int64_t nt = (int64_t)(blockIdx.x - cell_blocks) * BS_T + threadIdx.x;
    bool act = false;
    if (nt < V.total_nt) {
        const SceneDev& sc = V.scenes[scene_of_node_tile(V, (int)nt)];
        const int l = (int)nt - sc.nt_base;
        const int x = l % sc.nt[0], y = (l / sc.nt[0]) % sc.nt[1], z = l / (sc.nt[0] * sc.nt[1]);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int cx = x - (k & 1), cy = y - ((k >> 1) & 1), cz = z - (k >> 2);
            if (cx < 0 || cy < 0 || cz < 0 || cx >= sc.ct[0] || cy >= sc.ct[1] || cz >= sc.ct[2]) continue;
            act |= c.tcount[sc.ct_base + (cz * sc.ct[1] + cy) * sc.ct[0] + cx] > 0u;
        }
        V.tile_flags[nt] = act ? 1u : 0u;
    }
    bs_append(V.tile_list, &V.sort_work[SW_TILES], act, (uint32_t)nt, lane);
}

// Blocks [0, tile_blocks): the work list and the counters, the rest: the
// particles, whose sorted keys and indices go to ok_ and ov -- or (REC), from
// the caller's arrays of R, as records to the state planes: (u - s - 1, m)
// with u the grid coordinates and s the cell's lowest node, (v, index) and for
// the reverse (gv + dt gx, 0).
template <bool REC>
__global__ void __launch_bounds__(BS_T) bs_scatter(View V, const uint32_t* keys, SortCounts c, const uint2* cell_range,
                                                   const uint4* tile_info, uint4* ptile, uint32_t* ok_,
                                                   uint32_t* ov, int tile_blocks, RefStep R) {
    step_wait();
    const int64_t n = V.N;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if ((int)blockIdx.x < tile_blocks) {
        // the largest-first work list, and the counters cleared for the next sort
        const int gid = (int)blockIdx.x * BS_T + threadIdx.x, threads = tile_blocks * BS_T;
        const uint32_t ntiles = V.sort_work[SW_CTILES];
        uint32_t in_class[CNT_BUCKETS];
#pragma unroll
        for (int b = 0; b < CNT_BUCKETS; ++b) in_class[b] = V.sort_work[SW_BUCKET + b];
        for (uint32_t i = gid; i < ntiles; i += threads) {
            const uint4 t = tile_info[i];
            const uint32_t cls = t.w >> 28;
            uint32_t off = t.w & 0x0FFFFFFFu;
#pragma unroll
            for (uint32_t b = 0; b < (uint32_t)CNT_BUCKETS; ++b) off += b < cls ? in_class[b] : 0u;
            ptile[off] = make_uint4(t.x, t.y, t.z, (uint32_t)scene_of_cell_tile(V, (int)t.x));
            c.tcount[t.x] = 0u;
        }
        if (gid < CNT_RESET)
            V.counters[gid] = gid == CNT_TILES ? V.sort_work[SW_TILES] : gid == CNT_CTILES ? ntiles : 0u;
        if (gid == 0) {
            c.tcount[V.total_ct] = 0u;
            c.ccount[c.ncells] = 0u;
        }
        return;
    }
    constexpr int ITEMS = REC ? BS_REC_ITEMS : BS_ITEMS;
    const int64_t base = (int64_t)(blockIdx.x - tile_blocks) * (BS_T * ITEMS) + warp * (32 * ITEMS);
    uint32_t k[ITEMS], sl[ITEMS], pos[ITEMS];
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
        const int64_t i = base + r * 32 + lane;
        k[r] = i < n ? keys[i] : 0u;
        sl[r] = i < n ? c.slot[i] : 0u;
    }
#pragma unroll
    for (int r = 0; r < ITEMS; ++r)
        pos[r] = (k[r] < c.ncells ? cell_range[k[r]].x : V.sort_work[SW_VALID]) + sl[r];
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
        const int64_t i = base + r * 32 + lane;
        if (i < n && (int64_t)pos[r] < n) {
            if (REC) {
                const SceneDev& sc = V.scenes[0];
                float g[3];
                uint32_t f = 0;
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    float u;
                    const int s = stencil_origin(R.x[3 * i + a], sc.origin[a], sc.dx, sc.inv_dx, sc.n[a], PHYS_REF, u, f);
                    g[a] = __fsub_rn(u, (float)(s + 1));
                }
                V.q[pos[r]] = make_float4(g[0], g[1], g[2], R.m[i]);
                V.q[n + pos[r]] = make_float4(R.v[3 * i], R.v[3 * i + 1], R.v[3 * i + 2], __uint_as_float((uint32_t)i));
                if (R.gx) {
                    const float dt = sc.dt;
                    V.q[2 * n + pos[r]] = make_float4(R.gv[3 * i] + dt * R.gx[3 * i], R.gv[3 * i + 1] + dt * R.gx[3 * i + 1],
                                                      R.gv[3 * i + 2] + dt * R.gx[3 * i + 2], 0.f);
                }
            } else {
                ok_[pos[r]] = k[r];
                ov[pos[r]] = (uint32_t)i;
            }
        }
    }
}
}  // namespace

int64_t bin_sort_groups(int64_t total_ct) { return (total_ct + BS_GROUP) / BS_GROUP; }

cudaError_t bin_sort_step(const View& V, const BinSortBufs& B, int num_sms, bool counted, cudaStream_t st,
                          const RefStep* rec) {
    const int64_t n = V.N;
    if (n <= 0) return cudaSuccess;
    if (!B.cell_range || !B.ptile || !V.sort_work) return cudaErrorInvalidValue;
    const int gk = (int)((n + BS_TILE - 1) / BS_TILE);
    const int64_t nct = V.total_ct;
    cudaError_t e = cudaSuccess;
    if (!counted) e = launch_after(V.early_first, bs_count, gk, BS_T, st, B.keys_in, n, B.cnt, V.counters);
    bool early = counted ? V.early_first : V.early;
    const uint32_t* gsum = nct > BS_DIRECT_TILES ? B.gsum : nullptr;
    if (gsum && e == cudaSuccess) {
        e = launch_after(early, bs_groups, (int)bin_sort_groups(nct), BS_T, st, B.cnt.tcount, nct + 1, B.gsum);
        early = V.early;
    }
    if (e != cudaSuccess) return e;
    // sparse grids mark their node tiles from the occupied cell tiles
    const int node_blocks = V.sp.cap ? 0 : (V.total_nt + BS_T - 1) / BS_T;
    const int per_block = (nct <= BT_FEW_TILES ? BT_FEW : BT_MANY) * (BS_T / 32);
    const int cell_blocks = (int)((nct + per_block - 1) / per_block);
    e = launch_after(early, nct <= BT_FEW_TILES ? bs_tiles<BT_FEW> : bs_tiles<BT_MANY>, cell_blocks + node_blocks, BS_T,
                     st, V, B.cnt, gsum, B.cell_range, B.tile_info, cell_blocks);
    if (e != cudaSuccess) return e;
    const int tile_blocks = (int)std::min<int64_t>(num_sms, (nct + BS_T - 1) / BS_T);
    if (rec)
        return launch_after(V.early, bs_scatter<true>,
                            tile_blocks + (int)((n + BS_T * BS_REC_ITEMS - 1) / (BS_T * BS_REC_ITEMS)), BS_T, st, V,
                            B.keys_in, B.cnt, B.cell_range, B.tile_info, B.ptile, nullptr, nullptr, tile_blocks, *rec);
    return launch_after(V.early, bs_scatter<false>, tile_blocks + gk, BS_T, st, V, B.keys_in, B.cnt, B.cell_range,
                        B.tile_info, B.ptile, B.out_k, B.out_v, tile_blocks, RefStep{});
}

int64_t radix_sort_scratch_words(int64_t n) { return radix_scratch_words_for(n); }

int radix_passes(int key_bits) { return key_bits <= 0 ? 0 : (key_bits + 7) / 8; }

// Sorts (kin, vin) by the low key_bits bits.  Buffers: (ka, va), (kb, vb)
// ping-pong targets of n words each; scratch of radix_sort_scratch_words(n)
// u32.  Returns which buffer pair holds the result (0 = a, 1 = b) through
// *which.  vin may be null (values = index).  No allocation, no sync.
cudaError_t radix_sort_pairs(const uint32_t* kin, const uint32_t* vin, uint32_t* ka, uint32_t* va, uint32_t* kb,
                             uint32_t* vb, uint32_t* scratch, int64_t n, int key_bits, int* which,
                             cudaStream_t st) {
    *which = 0;
    if (n <= 0) return cudaSuccess;
    const int passes = radix_passes(key_bits < 1 ? 1 : key_bits);
    const int bits = (key_bits + passes - 1) / passes;
    const int nb = (int)((n + RS_TILE - 1) / RS_TILE);
    uint32_t* hist = scratch;
    uint32_t* totals = scratch + (int64_t)nb * RS_MAXD;
    const uint32_t* ck = kin;
    const uint32_t* cv = vin;
    int shift = 0;
    for (int p = 0; p < passes; ++p) {
        uint32_t* ok = (p & 1) ? kb : ka;
        uint32_t* ov = (p & 1) ? vb : va;
        const int b = min(bits, key_bits - shift) > 0 ? min(bits, key_bits - shift) : 1;
        cudaError_t e = launch_after(p > 0, rs_hist, nb, RS_THREADS, st, ck, n, shift, b, hist, nb);
        if (e == cudaSuccess) e = launch_after(true, rs_scan, 1 << b, 1024, st, hist, nb, totals);
        if (e == cudaSuccess)
            e = launch_after(true, rs_scatter, nb, RS_THREADS, st, ck, cv, ok, ov, n, shift, b, hist, nb, totals);
        if (e != cudaSuccess) return e;
        ck = ok;
        cv = ov;
        shift += b;
        *which = p & 1;
    }
    return cudaSuccess;
}

}  // namespace pgmpm
