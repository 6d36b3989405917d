// pgmpm_coupling.cu -- consumers of the solver's particles on the device:
//   * pgmpm_sph_coupling: the SPH-MPM contact coupling of
//     SPHMPMCouplingSystem (src/sph_mpm_coupling.h:453-575), with the
//     solver's particles as the MPM side.  The MPM particles are counted into
//     cells of half a coupling radius (the cell coordinates of the reference's
//     SpatialHashGrid, laid out in grid order) and their positions and
//     velocities copied into that order; one warp per SPH particle walks the
//     cells within one radius of it, keeps the pairs closer than the radius and
//     forms their forces in the reference's float operations, in the same
//     order, so pair membership is bit-exact; only the order in which a
//     particle's pair forces are summed differs.
//   * pgmpm_kinetic_energy: the energy monitor of FSISimulationManager
//     (computeTotalEnergy, src/fsi_coupling.h:837-858), per material.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "pgmpm_hashgrid.cuh"
#include "pgmpm_solver_impl.h"

using namespace pgmpm;

namespace {

// Cell of an MPM particle: the reference's cell coordinates, clamped to the
// grid, in grid order (x outer, z inner).
__device__ __forceinline__ uint32_t cpl_cell(const HGDev& G, const float4& x) {
    const uint32_t c0 = min(hg_coord(x.x, G.dmin[0], G.cell), G.res[0] - 1u),
                   c1 = min(hg_coord(x.y, G.dmin[1], G.cell), G.res[1] - 1u),
                   c2 = min(hg_coord(x.z, G.dmin[2], G.cell), G.res[2] - 1u);
    return (c0 * G.res[1] + c1) * G.res[2] + c2;
}
// particles per cell, and each particle's slot in its cell
__global__ void k_cpl_count(HGDev G, const float4* __restrict__ q, int64_t N, uint32_t* __restrict__ count,
                            uint32_t* __restrict__ slot) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < N; p += stride)
        slot[p] = atomicAdd(&count[cpl_cell(G, q[p])], 1u);
}
// x (with the particle's index) and v in cell order, the force sums cleared
__global__ void k_cpl_scatter(HGDev G, const float4* __restrict__ q, int64_t N, const uint32_t* __restrict__ first,
                              const uint32_t* __restrict__ slot, float4* __restrict__ xs, float4* __restrict__ vs,
                              float4* __restrict__ mf) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < N; p += stride) {
        const float4 x = q[p];
        const size_t i = first[cpl_cell(G, x)] + slot[p];
        xs[i] = make_float4(x.x, x.y, x.z, __uint_as_float((uint32_t)p));
        vs[i] = q[3 * N + p];
        if (mf) mf[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
}
// solid force sums (cell order) -> the caller's [N][3] array in upload order
__global__ void k_mforce_out(const float4* __restrict__ mf, const float4* __restrict__ xs,
                             const uint32_t* __restrict__ user_of_phys, int64_t N, float* __restrict__ out) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < N; i += stride) {
        const float4 f = mf[i];
        const size_t u = user_of_phys[__float_as_uint(xs[i].w)];
        out[3 * u] = f.x;
        out[3 * u + 1] = f.y;
        out[3 * u + 2] = f.z;
    }
}

// Margin, in cells, of the cut at cell coordinate g.  A coordinate is the
// rounded quotient of a rounded difference (2^-23 of it off), and a cell's face
// is formed with as much error again: 2^-22 g, the same for a bound of the z
// window.  1e-3 alone dropped one pair in a few thousand at the edge of the
// sphere from 60,000 cells an axis on.  The last sum and difference need none:
// rounding keeps the order of what the pair test rounds too.
__device__ __forceinline__ float cpl_margin(float g) { return 1e-3f + 0x1p-21f * g; }
// Distance from y to cell g along axis a, a lower bound for any particle stored
// there (the last cell also holds clamped particles: 0).
__device__ __forceinline__ float cpl_gap(const HGDev& G, int a, float y, uint32_t g) {
    const float m = cpl_margin((float)g);
    const float lo = G.dmin[a] + ((float)g - m) * G.cell, hi = G.dmin[a] + ((float)g + (1.f + m)) * G.cell;
    return g + 1u == G.res[a] ? 0.f : fmaxf(fmaxf(g == 0u ? 0.f : lo - y, y - hi), 0.f);
}
// hg_row cut to the cells that the sphere of radius r around y (cell c) can
// reach: of the 125 cells of half a radius each around a particle the sphere
// meets about 60%.  The margins (cpl_margin, and 1e-5 of r^2 for the rounding
// of the squared distances) are above the rounding, so that the cut drops no pair.
__device__ __forceinline__ uint2 cpl_row(const HGDev& G, const uint32_t c[3], uint32_t src, uint32_t dx, uint32_t dy,
                                         const float y[3], float r, const uint32_t* __restrict__ first) {
    const uint32_t gx = c[0] + dx - src, gy = c[1] + dy - src;
    if (gx >= G.res[0] || gy >= G.res[1]) return make_uint2(0u, 0u);
    const float a = cpl_gap(G, 0, y[0], gx), b = cpl_gap(G, 1, y[1], gy);
    const float z2 = r * r * 1.00001f - a * a - b * b;
    if (z2 < 0.f) return make_uint2(0u, 0u);
    const float zr = sqrtf(z2), inv = 1.f / G.cell;
    const float t0 = (y[2] - zr - G.dmin[2]) * inv, t1 = (y[2] + zr - G.dmin[2]) * inv;
    const float f0 = floorf(t0 - cpl_margin(fabsf(t0))), f1 = floorf(t1 + cpl_margin(fabsf(t1)));
    // the window [c2 - src, c2 + src] as signed 64-bit, cut at the sphere and the grid
    const long long z = (long long)(int)c[2], last = (long long)G.res[2] - 1;
    long long z0 = max(z - (long long)src, 0ll), z1 = min(z + (long long)src, last);
    if (f0 > (float)z0) z0 = (long long)fminf(f0, (float)last);
    if (f1 < (float)z1 && f1 >= 0.f) z1 = (long long)f1;
    if (z0 > z1) return make_uint2(0u, 0u);
    const uint32_t row = (gx * G.res[1] + gy) * G.res[2];
    const uint32_t f = __ldg(&first[row + (uint32_t)z0]);
    return make_uint2(f, __ldg(&first[row + (uint32_t)z1 + 1u]) - f);
}

// One warp per SPH particle: its candidates are the MPM particles of the cells
// within one radius, one stretch of the cell order per cell row along z; the
// lanes take them in turn, two at a time, so that a warp's candidate reads and
// force atomics run along memory.  d2_max: the smallest float whose square root
// is not below r, so that d^2 < d2_max holds for exactly the pairs with d < r.
// The pairs (a quarter of the candidates in a block of cells) are queued and
// processed 32 at a time, so that the force arithmetic runs on full warps: the
// contact force (normal spring and damping, friction along the tangential
// velocity), the fluid force, summed over the warp, to sph_force (two-way), the
// solid force to mforce (one vector atomic per pair), the pair count and
// k (r - d)^2 / 2 to npairs and energy.
//
// Bound by the candidates' tests (latency and instructions; the atomics take
// 4%).  1 M MPM and 131 K SPH particles, 96 M candidates, 29 M pairs: candidate
// lists from the neighbour query, gathered from the state planes, took 77 + 394
// us for the lists and 940 us for the pairs; the hash grid's cells walked in
// place 813 us (777 with the queue), grid-order stretches with two candidates
// in flight 622, cut to the cells the sphere meets 520 (cells of a third or a
// quarter radius: 526 and 564).
__global__ void __launch_bounds__(256) k_sph_pairs(HGDev G, const uint32_t* __restrict__ first, uint32_t src,
                                                   const float* __restrict__ sx, const float* __restrict__ sv,
                                                   int64_t nq, const float4* __restrict__ xs,
                                                   const float4* __restrict__ vs, float d2_max, bool cut,
                                                   pgmpm_sph_coupling_config cfg, float* __restrict__ sph_force,
                                                   float4* __restrict__ mforce, unsigned long long* __restrict__ npairs,
                                                   double* __restrict__ energy) {
    __shared__ float4 s_r[8][128];  // per warp: queued pairs (x_mpm - x_sph, distance squared)
    __shared__ uint32_t s_p[8][128];
    __shared__ uint32_t s_end[8][32], s_shift[8][32];  // per warp: the stretches as one list
    constexpr uint32_t FULL = 0xFFFFFFFFu;
    const uint32_t w = 2 * src + 1, nrow = w * w;
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    float4* const q_r = s_r[wp];
    uint32_t* const q_p = s_p[wp];
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    const float k = cfg.coupling_stiffness, c = cfg.coupling_damping, mu = cfg.friction_coefficient,
                r = cfg.coupling_radius;
    unsigned long long cnt = 0;
    double e = 0.0;
    for (int64_t q = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; q < nq; q += warps) {
        const float y0 = sx[3 * q], y1 = sx[3 * q + 1], y2 = sx[3 * q + 2];
        const float w0 = sv[3 * q], w1 = sv[3 * q + 1], w2 = sv[3 * q + 2];
        const uint32_t cc[3] = {hg_coord(y0, G.dmin[0], G.cell), hg_coord(y1, G.dmin[1], G.cell),
                                hg_coord(y2, G.dmin[2], G.cell)};
        float f0 = 0.f, f1 = 0.f, f2 = 0.f;
        uint32_t head = 0, tail = 0;  // queue of pairs: entries head .. tail - 1 (mod 128)
        auto pair = [&](uint32_t at) {
            const float4 rd = q_r[at];
            const uint32_t p = q_p[at];
            const float d = sqrtf(rd.w);
            ++cnt;
            const float pen = __fsub_rn(r, d);
            e += (double)__fmul_rn(__fmul_rn(__fmul_rn(0.5f, k), pen), pen);
            if (d < 1e-6f) return;
            const float inv = __fdiv_rn(1.f, d);
            const float n0 = __fmul_rn(rd.x, inv), n1 = __fmul_rn(rd.y, inv), n2 = __fmul_rn(rd.z, inv);
            const float4 vp = __ldg(&vs[p]);
            const float d0 = __fsub_rn(vp.x, w0), d1 = __fsub_rn(vp.y, w1), d2 = __fsub_rn(vp.z, w2);
            const float fn = __fmul_rn(k, pen);
            const float vn = __fadd_rn(__fadd_rn(__fmul_rn(d0, n0), __fmul_rn(d1, n1)), __fmul_rn(d2, n2));
            const float ft = __fadd_rn(fn, __fmul_rn(c, vn));
            float g0 = __fmul_rn(n0, ft), g1 = __fmul_rn(n1, ft), g2 = __fmul_rn(n2, ft);
            const float u0 = __fsub_rn(d0, __fmul_rn(n0, vn)), u1 = __fsub_rn(d1, __fmul_rn(n1, vn)),
                        u2 = __fsub_rn(d2, __fmul_rn(n2, vn));
            const float ts = sqrtf(__fadd_rn(__fadd_rn(__fmul_rn(u0, u0), __fmul_rn(u1, u1)), __fmul_rn(u2, u2)));
            if (ts > 1e-6f) {
                const float it = __fdiv_rn(1.f, ts), fm = -__fmul_rn(mu, fn);
                g0 = __fadd_rn(g0, __fmul_rn(__fmul_rn(u0, it), fm));
                g1 = __fadd_rn(g1, __fmul_rn(__fmul_rn(u1, it), fm));
                g2 = __fadd_rn(g2, __fmul_rn(__fmul_rn(u2, it), fm));
            }
            f0 = __fadd_rn(f0, -g0);
            f1 = __fadd_rn(f1, -g1);
            f2 = __fadd_rn(f2, -g2);
            if (mforce) atomicAdd(&mforce[p], make_float4(g0, g1, g2, 0.f));
        };
        for (uint32_t t0 = 0; t0 < nrow; t0 += 32) {
            uint2 seg = make_uint2(0u, 0u);
            if (t0 + lane < nrow) {
                const uint32_t dx = (t0 + lane) / w, dy = (t0 + lane) % w;
                const float y[3] = {y0, y1, y2};
                seg = cut ? cpl_row(G, cc, src, dx, dy, y, r, first) : hg_row(G, cc, src, dx, dy, first);
            }
            uint32_t x = seg.y;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(FULL, x, o);
                if (lane >= o) x += y;
            }
            const uint32_t total = __shfl_sync(FULL, x, 31);
            __syncwarp();
            s_end[wp][lane] = x;
            s_shift[wp][lane] = seg.x - (x - seg.y);  // position = entry + shift of its stretch
            __syncwarp();
            int at = 0;  // this lane's stretch: the entries it takes come in order
            for (uint32_t e0 = 0; e0 < total; e0 += 64) {
                float4 cand[2];
                uint32_t pos[2];
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const uint32_t i = e0 + 32 * u + lane;
                    pos[u] = FULL;
                    if (i < total) {
                        while (i >= s_end[wp][at]) ++at;
                        pos[u] = i + s_shift[wp][at];
                        cand[u] = __ldg(&xs[pos[u]]);
                    }
                }
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    // distance as the reference forms it (no contraction)
                    float r0 = 0.f, r1 = 0.f, r2 = 0.f, d2 = d2_max;
                    if (pos[u] != FULL) {
                        r0 = __fsub_rn(cand[u].x, y0);
                        r1 = __fsub_rn(cand[u].y, y1);
                        r2 = __fsub_rn(cand[u].z, y2);
                        d2 = __fadd_rn(__fadd_rn(__fmul_rn(r0, r0), __fmul_rn(r1, r1)), __fmul_rn(r2, r2));
                    }
                    const uint32_t hit = __ballot_sync(FULL, d2 < d2_max);
                    if (d2 < d2_max) {
                        const uint32_t to = (tail + __popc(hit & ((1u << lane) - 1u))) & 127u;
                        q_r[to] = make_float4(r0, r1, r2, d2);
                        q_p[to] = pos[u];
                    }
                    tail += __popc(hit);
                }
                __syncwarp();
                while (tail - head >= 32u) {
                    pair((head + lane) & 127u);
                    head += 32u;
                }
                __syncwarp();
            }
        }
        if ((uint32_t)lane < tail - head) pair((head + lane) & 127u);
        __syncwarp();
        if (cfg.enable_two_way_coupling) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                f0 += __shfl_down_sync(0xFFFFFFFFu, f0, o);
                f1 += __shfl_down_sync(0xFFFFFFFFu, f1, o);
                f2 += __shfl_down_sync(0xFFFFFFFFu, f2, o);
            }
            if (lane == 0) {
                sph_force[3 * q] += f0;
                sph_force[3 * q + 1] += f1;
                sph_force[3 * q + 2] += f2;
            }
        }
    }
    // warp sums of the pair count and the energy, one atomic each per warp
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        cnt += __shfl_down_sync(0xFFFFFFFFu, cnt, o);
        e += __shfl_down_sync(0xFFFFFFFFu, e, o);
    }
    if (lane == 0) {
        if (cnt) atomicAdd(npairs, cnt);
        if (e != 0.0) atomicAdd(energy, e);
    }
}

// Per-material sums of m |v|^2 / 2 in FP64.  Up to KE_REG_MATS materials each
// thread keeps one register sum per material, and each warp adds its sums
// with one atomic per material; with more, per-block shared-memory sums take
// the particles' terms.  (One global atomic per particle on a handful of
// addresses serialises: 3 ms for 2 M particles of two materials.)
constexpr int KE_REG_MATS = 8;
constexpr int KE_SMEM_MATS = 64;
template <int MR>
__global__ void k_kinetic(const float4* __restrict__ q, const float2* __restrict__ mV, const int32_t* __restrict__ mat,
                          int64_t N, int M, double* __restrict__ out) {
    __shared__ double s_acc[KE_SMEM_MATS];
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    double acc[MR > 0 ? MR : 1];
#pragma unroll
    for (int m = 0; m < (MR > 0 ? MR : 1); ++m) acc[m] = 0.0;
    if (MR == 0) {
        for (int m = threadIdx.x; m < KE_SMEM_MATS; m += blockDim.x) s_acc[m] = 0.0;
        __syncthreads();
    }
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < N; p += stride) {
        const float4 v = q[3 * N + p];
        const double ke = 0.5 * (double)mV[p].x * ((double)v.x * v.x + (double)v.y * v.y + (double)v.z * v.z);
        const int id = mat ? min(max(mat[p], 0), M - 1) : 0;
        if (MR > 0) {
#pragma unroll
            for (int m = 0; m < (MR > 0 ? MR : 1); ++m) acc[m] += id == m ? ke : 0.0;
        } else if (M <= KE_SMEM_MATS) {
            atomicAdd(&s_acc[id], ke);
        } else {
            atomicAdd(&out[id], ke);
        }
    }
    if (MR > 0) {
#pragma unroll
        for (int m = 0; m < (MR > 0 ? MR : 1); ++m) {
            double e = acc[m];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) e += __shfl_down_sync(0xFFFFFFFFu, e, o);
            if ((threadIdx.x & 31) == 0 && e != 0.0 && m < M) atomicAdd(&out[m], e);
        }
    } else if (M <= KE_SMEM_MATS) {
        __syncthreads();
        for (int m = threadIdx.x; m < M; m += blockDim.x)
            if (s_acc[m] != 0.0) atomicAdd(&out[m], s_acc[m]);
    }
}

int nblocks(int64_t n, int t, int cap) { return (int)std::max<int64_t>(1, std::min<int64_t>((n + t - 1) / t, cap)); }

}  // namespace

extern "C" {

int pgmpm_sph_coupling(pgmpm_solver s, const pgmpm_sph_coupling_config* cfg, const float* sph_x, const float* sph_v,
                       int64_t n_sph, float* sph_force, float* mpm_force, int64_t* n_pairs, double* energy,
                       int32_t ptr_kind, void* stream) {
    if (!s || !cfg || n_sph < 0) return fail(PGMPM_ERR_ARG, "pgmpm_sph_coupling: bad arguments");
    if (!s->uploaded) return fail(PGMPM_ERR_STATE, "no particles uploaded");
    if (s->S != 1) return fail(PGMPM_ERR_UNSUPPORTED, "pgmpm_sph_coupling: one scene");
    if (!(cfg->coupling_radius > 0.f) || !std::isfinite(cfg->coupling_radius))
        return fail(PGMPM_ERR_ARG, "pgmpm_sph_coupling: coupling_radius must be positive");
    if (n_sph > 0 && (!sph_x || !sph_v || (cfg->enable_two_way_coupling && !sph_force)))
        return fail(PGMPM_ERR_ARG, "pgmpm_sph_coupling: sph_x, sph_v (and sph_force when two-way) are required");
    if (ptr_kind != PGMPM_PTR_HOST && ptr_kind != PGMPM_PTR_DEVICE) return fail(PGMPM_ERR_ARG, "bad ptr_kind");
    DeviceGuard dg(s->device);
    cudaStream_t st = ST(stream);
    const int64_t N = s->N;
    const size_t Nz = (size_t)std::max<int64_t>(N, 1), Qz = (size_t)std::max<int64_t>(n_sph, 1);
    // the SPH side on the device
    const float *dsx = sph_x, *dsv = sph_v;
    float* dsf = sph_force;
    float* dmf = mpm_force;
    if (ptr_kind == PGMPM_PTR_HOST) {
        CK(s->cpl_stage.ensure(sizeof(float) * (9 * Qz + 3 * Nz)));
        float* b = s->cpl_stage.as<float>();
        if (n_sph > 0) {
            CK(cudaMemcpyAsync(b, sph_x, sizeof(float) * 3 * n_sph, cudaMemcpyHostToDevice, st));
            CK(cudaMemcpyAsync(b + 3 * Qz, sph_v, sizeof(float) * 3 * n_sph, cudaMemcpyHostToDevice, st));
            if (cfg->enable_two_way_coupling)
                CK(cudaMemcpyAsync(b + 6 * Qz, sph_force, sizeof(float) * 3 * n_sph, cudaMemcpyHostToDevice, st));
        }
        dsx = b;
        dsv = b + 3 * Qz;
        dsf = b + 6 * Qz;
        dmf = mpm_force ? b + 9 * Qz : nullptr;
    }
    // x, v and the solid forces in cell order
    CK(s->cpl_mf.ensure(sizeof(float4) * 3 * Nz));
    float4 *xs = s->cpl_mf.as<float4>(), *vs = xs + Nz, *mf = dmf ? xs + 2 * Nz : nullptr;
    CK(s->cpl_acc.ensure(sizeof(double) * 2));
    CK(cudaMemsetAsync(s->cpl_acc.p, 0, sizeof(double) * 2, st));
    unsigned long long* d_pairs = s->cpl_acc.as<unsigned long long>();
    double* d_energy = s->cpl_acc.as<double>() + 1;
    if (N > 0 && n_sph > 0) {
        // the cell grid over the scene's domain.  Cells of half a
        // radius (125 around a particle) hold 42% fewer candidates than cells
        // of one radius (27), unless that makes more than 4 cells per MPM
        // particle (or 2^20, if more).
        const pgmpm_scene_desc& d = s->desc[0];
        float lo[3], hi[3];
        for (int a = 0; a < 3; ++a) {
            lo[a] = d.origin[a];
            hi[a] = d.origin[a] + (float)(d.n[a] - 1) * d.dx;
        }
        double cells_half = 1.0;
        for (int a = 0; a < 3; ++a) cells_half *= std::ceil((hi[a] - lo[a]) / (0.5 * cfg->coupling_radius));
        const float cell = cells_half <= std::max(4.0 * (double)N, (double)(1 << 20)) ? 0.5f * cfg->coupling_radius
                                                                                      : cfg->coupling_radius;
        HGDev G{};
        G.cell = cell;
        uint64_t total = 1;
        for (int a = 0; a < 3; ++a) {
            G.dmin[a] = lo[a];
            const float n = std::ceil((hi[a] - lo[a]) / cell);  // single precision, as pgmpm_hashgrid_create
            if (!(n >= 1.f) || !(n < 4294967296.f))
                return fail(PGMPM_ERR_ARG, "hashgrid: each axis needs 1 .. 2^32-1 cells");
            G.res[a] = (uint32_t)n;
            total *= G.res[a];
            if (total > 0xFFFFFFFFull) return fail(PGMPM_ERR_ARG, "hashgrid: more than 2^32 - 1 cells");
        }
        const float sr = std::ceil(cfg->coupling_radius / cell);  // cells a radius spans
        float d2_max = cfg->coupling_radius * cfg->coupling_radius;
        while (d2_max > 0.f && std::sqrt(d2_max) >= cfg->coupling_radius) d2_max = std::nextafter(d2_max, 0.f);
        while (std::sqrt(d2_max) < cfg->coupling_radius) d2_max = std::nextafter(d2_max, INFINITY);
        // few cells: a block may reach the last cell, which also holds particles
        // clamped from below, from the first ones
        const bool cut = std::min({G.res[0], G.res[1], G.res[2]}) > 8u + 2u * (uint32_t)sr;
        // counts (then each particle's slot after them), first[], block sums
        const size_t scan_bytes = exclusive_scan_bytes((int64_t)total);
        CK(s->cpl_cells.ensure(sizeof(uint32_t) * (2 * total + 2 + (size_t)N) + scan_bytes));
        int64_t* scan = s->cpl_cells.as<int64_t>();
        uint32_t* count = reinterpret_cast<uint32_t*>(s->cpl_cells.as<char>() + scan_bytes);
        uint32_t *first = count + total, *slot = first + total + 1;
        CK(cudaMemsetAsync(count, 0, sizeof(uint32_t) * total, st));
        const int nb = nblocks(N, 256, 148 * 16);
        k_cpl_count<<<nb, 256, 0, st>>>(G, s->q.as<float4>(), N, count, slot);
        CK(exclusive_scan(count, (int64_t)total, scan, first, st));
        k_cpl_scatter<<<nb, 256, 0, st>>>(G, s->q.as<float4>(), N, first, slot, xs, vs, mf);
        k_sph_pairs<<<nblocks(n_sph * 32, 256, 148 * 16), 256, 0, st>>>(G, first, (uint32_t)sr, dsx, dsv, n_sph, xs, vs,
                                                                        d2_max, cut, *cfg, dsf, mf, d_pairs, d_energy);
        if (mf)
            k_mforce_out<<<nblocks(N, 256, 148 * 16), 256, 0, st>>>(mf, xs, s->user_of_phys.as<uint32_t>(), N,
                                                                    dmf);
    } else if (dmf && N > 0) {
        CK(cudaMemsetAsync(dmf, 0, sizeof(float) * 3 * N, st));
    }
    CK(cudaGetLastError());
    if (ptr_kind == PGMPM_PTR_HOST) {
        if (cfg->enable_two_way_coupling && n_sph > 0)
            CK(cudaMemcpyAsync(sph_force, dsf, sizeof(float) * 3 * n_sph, cudaMemcpyDeviceToHost, st));
        if (mpm_force && N > 0) CK(cudaMemcpyAsync(mpm_force, dmf, sizeof(float) * 3 * N, cudaMemcpyDeviceToHost, st));
    }
    // pair count and energy in one read through pinned memory
    static_assert(2 * sizeof(double) <= CNT_WORDS * sizeof(uint32_t), "the counters' pinned words take both");
    CK(cudaMemcpyAsync(s->h_counters, s->cpl_acc.p, 2 * sizeof(double), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    unsigned long long h_pairs = 0;
    double h_energy = 0.0;
    std::memcpy(&h_pairs, s->h_counters, sizeof(h_pairs));
    std::memcpy(&h_energy, reinterpret_cast<const char*>(s->h_counters) + sizeof(double), sizeof(h_energy));
    if (n_pairs) *n_pairs = (int64_t)h_pairs;
    if (energy) *energy = h_energy;
    return PGMPM_OK;
}

int pgmpm_kinetic_energy(pgmpm_solver s, double* per_material, double* total, void* stream) {
    if (!s) return fail(PGMPM_ERR_ARG, "null solver");
    if (!s->uploaded) return fail(PGMPM_ERR_STATE, "no particles uploaded");
    DeviceGuard dg(s->device);
    cudaStream_t st = ST(stream);
    const int M = s->M;
    CK(s->cpl_acc.ensure(sizeof(double) * std::max(2, M)));
    CK(cudaMemsetAsync(s->cpl_acc.p, 0, sizeof(double) * M, st));
    if (s->N > 0) {
        const int nb = nblocks(s->N, 256, 148 * 8);
        const int32_t* mt = s->pf.multi_mat ? s->mat.as<int32_t>() : nullptr;
        if (!mt)
            k_kinetic<1><<<nb, 256, 0, st>>>(s->q.as<float4>(), s->mV.as<float2>(), nullptr, s->N, M,
                                             s->cpl_acc.as<double>());
        else if (M <= 2)
            k_kinetic<2><<<nb, 256, 0, st>>>(s->q.as<float4>(), s->mV.as<float2>(), mt, s->N, M,
                                             s->cpl_acc.as<double>());
        else if (M <= KE_REG_MATS)
            k_kinetic<KE_REG_MATS><<<nb, 256, 0, st>>>(s->q.as<float4>(), s->mV.as<float2>(), mt, s->N, M,
                                                       s->cpl_acc.as<double>());
        else
            k_kinetic<0><<<nb, 256, 0, st>>>(s->q.as<float4>(), s->mV.as<float2>(), mt, s->N, M,
                                             s->cpl_acc.as<double>());
    }
    CK(cudaGetLastError());
    std::vector<double> h(M);
    CK(cudaMemcpyAsync(h.data(), s->cpl_acc.p, sizeof(double) * M, cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    double t = 0.0;
    for (int i = 0; i < M; ++i) {
        if (per_material) per_material[i] = h[i];
        t += h[i];
    }
    if (total) *total = t;
    return PGMPM_OK;
}

}  // extern "C"
