// pgmpm_hashgrid.cuh -- device side of the spatial hash grid, shared by its own
// kernels (pgmpm_hashgrid.cu) and the contact coupling (pgmpm_coupling.cu).
// Not installed.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/pgmpm.h"

namespace pgmpm {

struct HGDev {
    float cell, dmin[3];
    uint32_t res[3], total;
    unsigned long long total_m;  // 2^64 / total + 1 (mod 2^64), for hg_mod
};

// a % total by direct computation of the remainder (Lemire, Kaser and Kurz,
// "Faster remainder by direct computation", 2019): for 32-bit a and d and
// M = floor(2^64 / d) + 1, a mod d = floor(((M a) mod 2^64) d / 2^64).
__device__ __forceinline__ uint32_t hg_mod(uint32_t a, const HGDev& G) {
    return (uint32_t)__umul64hi(G.total_m * (unsigned long long)a, (unsigned long long)G.total);
}

// src/sparse_data_structures.h:121-128: bit interleave in uint32 arithmetic
__device__ __forceinline__ uint32_t hg_expand(uint32_t v) {
    v = (v * 0x00010001u) & 0xFF0000FFu;
    v = (v * 0x00000101u) & 0x0F00F00Fu;
    v = (v * 0x00000011u) & 0xC30C30C3u;
    v = (v * 0x00000005u) & 0x49249249u;
    return v;
}
__device__ __forceinline__ uint32_t hg_morton(uint32_t x, uint32_t y, uint32_t z) {
    return hg_expand(x) | (hg_expand(y) << 1) | (hg_expand(z) << 2);
}
// (x - min) / cell in IEEE single, truncated toward zero to a 64-bit integer
// and reduced mod 2^32: the host's float -> uint32 conversion
__device__ __forceinline__ uint32_t hg_coord(float x, float mn, float cell) {
    return (uint32_t)(unsigned long long)__float2ll_rz(__fdiv_rn(__fsub_rn(x, mn), cell));
}

// (dx, dy, dz) of cell t of the block, packed 10 bits each, for the block's
// cells in shared memory when there are at most HG_TAB of them
constexpr int HG_TAB = 1024;
__device__ __forceinline__ uint32_t hg_offsets(uint32_t t, uint32_t w) {
    return (t % w) << 20 | ((t / w) % w) << 10 | (t / (w * w));
}
__device__ __forceinline__ void hg_fill_table(uint32_t* tab, uint32_t ncell, uint32_t w) {
    if (ncell <= (uint32_t)HG_TAB)
        for (uint32_t t = threadIdx.x; t < ncell; t += blockDim.x) tab[t] = hg_offsets(t, w);
    __syncthreads();
}
__device__ __forceinline__ bool hg_cell_of(const HGDev& G, const uint32_t c[3], uint32_t src, uint32_t w,
                                           uint32_t ncell, const uint32_t* tab, uint32_t t, uint32_t& id) {
    const uint32_t o = ncell <= (uint32_t)HG_TAB ? tab[t] : hg_offsets(t, w);
    const uint32_t dx = o & 1023u, dy = (o >> 10) & 1023u, dz = o >> 20;
    const uint32_t gx = c[0] + dx - src, gy = c[1] + dy - src, gz = c[2] + dz - src;  // wrap: below 0 fails
    if (gx >= G.res[0] || gy >= G.res[1] || gz >= G.res[2]) return false;
    id = hg_mod(hg_morton(gx, gy, gz), G);
    return true;
}

// With every cell's particles stored in grid order (x outer, z inner) from
// first[cell] on: the stretch (begin, length) of the cells of row (dx, dy) of
// the block of half width src around cell coordinates c.  c may be outside the
// grid (uint32 wrap: below 0 fails the range tests).
__device__ __forceinline__ uint2 hg_row(const HGDev& G, const uint32_t c[3], uint32_t src, uint32_t dx, uint32_t dy,
                                        const uint32_t* __restrict__ first) {
    const uint32_t gx = c[0] + dx - src, gy = c[1] + dy - src;
    if (gx >= G.res[0] || gy >= G.res[1]) return make_uint2(0u, 0u);
    // the z window [c2 - src, c2 + src] as signed 64-bit, cut at the grid
    const long long z = (long long)(int)c[2];
    const long long z0 = max(z - (long long)src, 0ll), z1 = min(z + (long long)src, (long long)G.res[2] - 1);
    if (z0 > z1) return make_uint2(0u, 0u);
    const uint32_t row = (gx * G.res[1] + gy) * G.res[2];
    const uint32_t f = __ldg(&first[row + (uint32_t)z0]);
    return make_uint2(f, __ldg(&first[row + (uint32_t)z1 + 1u]) - f);
}

// Exclusive scan of n counts into out[0..n] (out[n] = total, which may wrap;
// *total in 64 bits where asked for); scratch of exclusive_scan_bytes(n).
size_t exclusive_scan_bytes(int64_t n);
cudaError_t exclusive_scan(const uint32_t* in, int64_t n, int64_t* scratch, uint32_t* out, cudaStream_t st,
                           int64_t* total = nullptr);

// Walks the entries of up to 32 segments (start s0 and length k of this lane's
// segment, k = 0 for none) as one list, the warp's lanes taking consecutive
// entries: fn(valid, e, pos), called by the whole warp, for entry e of the list
// at position pos (valid: there is one for this lane).  A lane finds its
// entry's segment by a binary search over the lanes' inclusive lengths.
// Returns the list's length.
template <class Fn>
__device__ __forceinline__ uint32_t hg_walk(uint32_t s0, uint32_t k, int lane, const Fn& fn) {
    constexpr uint32_t FULL = 0xFFFFFFFFu;
    uint32_t x = k;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(FULL, x, o);
        if (lane >= o) x += y;
    }
    const uint32_t total = __shfl_sync(FULL, x, 31);
    const uint32_t shift = s0 - (x - k);  // position = entry + shift of its segment
    for (uint32_t e0 = 0; e0 < total; e0 += 32) {
        const uint32_t e = e0 + lane;
        int c = 0;  // first lane whose inclusive length exceeds e
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            if (__shfl_sync(FULL, x, c + o - 1) <= e) c += o;
        const uint32_t sh = __shfl_sync(FULL, shift, c & 31);
        fn(e < total, e, e + sh);
    }
    return total;
}

}  // namespace pgmpm
