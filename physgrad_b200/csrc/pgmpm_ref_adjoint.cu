// pgmpm_ref_adjoint.cu -- reverse of one REF_COMPAT step (the reference's PIC
// step, src/material_point_method.h:479-666) for launch_mpm_timestep_backward
// (src/pytorch_autograd.cu:384-402).
//
// Forward (per particle p, node i, REF weights w_pi of x_p, thresholded at
// 1e-10 and cut at the grid bounds):
//   m_i = sum_p w m_p,  P_i = sum_p w m_p v_p
//   v_i = (P_i + m_i g dt) / m_i = P_i / m_i + g dt     (m_i > 1e-10, else 0)
//   v'_p = sum_i w v_i,  x'_p = x_p + dt v'_p
// Reverse, given gx' = dL/dx', gv' = dL/dv':
//   1. k_ref_adj_scatter  a_p = gv' + dt gx';  Gv_i += w a_p
//   2. k_ref_adj_grid     gP_i = Gv_i / m_i, gm_i = -Gv_i . (P_i / m_i) / m_i,
//                         dL/dg += dt sum_i Gv_i
//   3. k_ref_adj_gather   dL/dx = gx' + sum_i grad w (a_p . v_i + m_p gm_i + m_p gP_i . v_p)
//                         dL/dv = sum_i w m_p gP_i
//                         dL/dm = sum_i w (gm_i + gP_i . v_p)
// Particles are read in the caller's order (upload order); the grid is the
// solver's tiled grid after the recomputed forward step.
//
// launch_ref_step runs a whole launch_mpm_timestep_forward or _backward call on
// the caller's arrays, for solvers with the bin sort: the particles are
// counted into cells and the sort's scatter writes their records (x, m, v and
// the reverse's gv' + dt gx') in sorted order; P2G and the reverse scatter run
// in one kernel (three threads per cell, one per z-offset, as the MLS P2G), and
// G2P and the reverse gather in the sorted order, where neighbouring threads
// share grid nodes.  Such a call is bound by
// its launches (100,003 particles on 64^3 nodes: 3-26 us each), so it makes
// six: no upload (a sort of three radix passes, a pack), no download, and in
// the backward no G2P.  A forward and a backward of 100,003 particles through
// autograd.MPMTimestep, 87 launches and 455 us of kernels before (486 us a pass
// with the one-pass upload), are 13 launches and 108 us (173 us a pass, bound by
// the host).  The records hold u - s - 1 so that P2G divides nothing (19
// against 24 us for P2G, 27 against 37 with the reverse scatter).
#include <algorithm>

#include "pgmpm_internal.h"

namespace pgmpm {
namespace {

// d/dr of the reference quadratic B-spline (ref_quadratic)
__device__ __forceinline__ float ref_quadratic_d(float r) {
    const float a = r < 0.f ? -r : r;
    if (a >= 1.5f) return 0.f;
    if (a < 0.5f) return -2.f * r;
    const float t = 1.5f - a;
    return r < 0.f ? t : -t;
}

// REF stencil of x with the weight derivatives (d/dx, per axis and node)
struct RefStencil {
    Stencil st;
    float dw[3][3];
};

__device__ __forceinline__ void ref_stencil(const SceneDev& sc, const float x[3], RefStencil& r, uint32_t& flags) {
    make_stencil<PHYS_REF>(sc, x, r.st, flags);
    const float idx = 1.f / sc.dx;
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int k = 0; k < 3; ++k) r.dw[a][k] = ref_quadratic_d(r.st.f[a] - (float)(k - 1)) * idx;
}

__global__ void k_ref_adj_scatter(View V, const float* __restrict__ x, const float* __restrict__ gx,
                                  const float* __restrict__ gv, float4* __restrict__ G, int64_t n) {
    const SceneDev& sc = V.scenes[0];
    uint32_t flags = 0;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += stride) {
        const float xp[3] = {x[3 * p], x[3 * p + 1], x[3 * p + 2]};
        Stencil st;
        make_stencil<PHYS_REF>(sc, xp, st, flags);
        float a[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) a[c] = gv[3 * p + c] + sc.dt * gx[3 * p + c];
#pragma unroll
        for (int ii = 0; ii < 3; ++ii) {
            const int gi = st.b[0] + ii;
            if (gi < 0 || gi >= sc.n[0]) continue;
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                const int gj = st.b[1] + j;
                if (gj < 0 || gj >= sc.n[1]) continue;
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const int gk = st.b[2] + k;
                    if (gk < 0 || gk >= sc.n[2]) continue;
                    const float w = __fmul_rn(__fmul_rn(st.w[0][ii], st.w[1][j]), st.w[2][k]);
                    if (!(w > 1e-10f)) continue;
                    float* g = reinterpret_cast<float*>(&G[node_index(sc, gi, gj, gk)]);
                    atomicAdd(g, w * a[0]);
                    atomicAdd(g + 1, w * a[1]);
                    atomicAdd(g + 2, w * a[2]);
                }
            }
        }
    }
}

// over the step's active node tiles (the only nodes a stencil reaches)
__global__ void k_ref_adj_grid(View V, float4* __restrict__ G, float* __restrict__ ggrav) {
    const SceneDev& sc = V.scenes[0];
    const uint32_t count = V.counters[CNT_TILES];
    const int tiles_per_block = blockDim.x >> 6;
    const int l = threadIdx.x & 63;
    float acc[3] = {0.f, 0.f, 0.f};
    for (uint32_t w = blockIdx.x * tiles_per_block + (threadIdx.x >> 6); w < count;
         w += gridDim.x * tiles_per_block) {
        const uint32_t nt = V.tile_list[w];
        if (nt >= (uint32_t)V.total_nt) continue;
        const int64_t idx = ((int64_t)nt << 6) + l;
        const float4 g = G[idx];
        const float4 vm = V.grid_v[idx];  // (v, m) of the forward step
        float4 out = make_float4(0.f, 0.f, 0.f, 0.f);
        if (vm.w > 1e-10f) {
            const float im = 1.f / vm.w;
            const float pm0 = vm.x - sc.gravity[0] * sc.dt, pm1 = vm.y - sc.gravity[1] * sc.dt,
                        pm2 = vm.z - sc.gravity[2] * sc.dt;  // P / m
            out = make_float4(g.x * im, g.y * im, g.z * im, -(g.x * pm0 + g.y * pm1 + g.z * pm2) * im);
            acc[0] += g.x;
            acc[1] += g.y;
            acc[2] += g.z;
        }
        G[idx] = out;
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        float s = acc[c] * sc.dt;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xFFFFFFFFu, s, o);
        if (ggrav && (threadIdx.x & 31) == 0 && s != 0.f) atomicAdd(&ggrav[c], s);
    }
}

__global__ void k_ref_adj_gather(View V, const float* __restrict__ x, const float* __restrict__ v,
                                 const float* __restrict__ m, const float* __restrict__ gx,
                                 const float* __restrict__ gv, const float4* __restrict__ G,
                                 float* __restrict__ gx_in, float* __restrict__ gv_in, float* __restrict__ gm_in,
                                 int64_t n) {
    const SceneDev& sc = V.scenes[0];
    uint32_t flags = 0;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += stride) {
        const float xp[3] = {x[3 * p], x[3 * p + 1], x[3 * p + 2]};
        const float vp[3] = {v[3 * p], v[3 * p + 1], v[3 * p + 2]};
        const float mp = m[p];
        RefStencil r;
        ref_stencil(sc, xp, r, flags);
        float a[3], ox[3], ov[3] = {0.f, 0.f, 0.f}, om = 0.f;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            ox[c] = gx[3 * p + c];
            a[c] = gv[3 * p + c] + sc.dt * ox[c];
        }
#pragma unroll
        for (int ii = 0; ii < 3; ++ii) {
            const int gi = r.st.b[0] + ii;
            if (gi < 0 || gi >= sc.n[0]) continue;
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                const int gj = r.st.b[1] + j;
                if (gj < 0 || gj >= sc.n[1]) continue;
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const int gk = r.st.b[2] + k;
                    if (gk < 0 || gk >= sc.n[2]) continue;
                    const float wx = r.st.w[0][ii], wy = r.st.w[1][j], wz = r.st.w[2][k];
                    const float w = __fmul_rn(__fmul_rn(wx, wy), wz);
                    if (!(w > 1e-10f)) continue;
                    const int64_t idx = node_index(sc, gi, gj, gk);
                    const float4 vi = V.grid_v[idx];
                    const float4 g = G[idx];  // (gP, gm)
                    const float gPv = g.x * vp[0] + g.y * vp[1] + g.z * vp[2];
                    const float s = a[0] * vi.x + a[1] * vi.y + a[2] * vi.z + mp * (g.w + gPv);
                    ox[0] += r.dw[0][ii] * wy * wz * s;
                    ox[1] += wx * r.dw[1][j] * wz * s;
                    ox[2] += wx * wy * r.dw[2][k] * s;
                    ov[0] += w * mp * g.x;
                    ov[1] += w * mp * g.y;
                    ov[2] += w * mp * g.z;
                    om += w * (g.w + gPv);
                }
            }
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            if (gx_in) gx_in[3 * p + c] = ox[c];
            if (gv_in) gv_in[3 * p + c] = ov[c];
        }
        if (gm_in) gm_in[p] = om;
    }
}

// ---------------------------------------- whole steps on the caller's arrays
// Keys of the caller's positions, counted for the bin sort; keeps the masses
// and the gravity for a later backward.
__global__ void __launch_bounds__(256) k_ref_keys(View V, RefStep R) {
    SceneDev* sc = const_cast<SceneDev*>(V.scenes);
    if (R.gravity && blockIdx.x == 0 && threadIdx.x < 3) sc->gravity[threadIdx.x] = R.gravity[threadIdx.x];
    uint32_t flags = 0;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < V.N; p += stride) {
        int so[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            float u;
            so[a] = stencil_origin(R.x[3 * p + a], sc->origin[a], sc->dx, sc->inv_dx, sc->n[a], PHYS_REF, u, flags);
        }
        const uint32_t key = cell_key(*sc, so);
        const KeyRun run = count_key(V.cnt, key);
        V.keys[p] = key;
        if (R.keep_m != R.m) R.keep_m[p] = R.m[p];
        V.cnt.slot[p] = run_slot(run);
    }
    if (flags) atomicOr(&V.counters[CNT_FLAGS], flags);
}

// Weights of a cell's nodes s .. s + 2 along one axis for a particle at g = u -
// s - 1: those of its own stencil's nodes (floor(u) - 1 .. floor(u) + 1), zero
// for a node it does not reach (a stencil that the grid's faces cut).
__device__ __forceinline__ float ref_cell_weight(float g, int o) {
    const int idx = o - (int)fminf(fmaxf(floorf(g), -8.f), 8.f);  // the node's place in the particle's stencil
    return (unsigned)idx <= 2u ? ref_quadratic(__fsub_rn(g, (float)(o - 1))) : 0.f;
}

// P2G of the step; ADJ: and the reverse of its G2P (a = gv' + dt gx' onto
// R.acc), whose weights are the same.
template <bool ADJ>
__global__ void __launch_bounds__(P2GS_T, ADJ ? 3 : 4) k_ref_p2g(View V, RefStep R) {
    __shared__ float4 T4[3 * P2GS_PLANE];
    const int t = threadIdx.x;
    const int q = t / 3, k = t - 3 * (t / 3);
    const SceneDev& sc = V.scenes[0];
    const uint32_t ntiles = V.counters[CNT_CTILES];
    // slices of a cell's particles when tiles are few.  Rounded up, at most 4,
    // where k_p2g_slices rounds down, to 8: items go to the blocks in turn here,
    // without claims (median of forward and reverse, that rule after this one:
    // 200,000 particles on 40^3 nodes 29.1 and 30.1 us, 10,000 on 32^3 11.0 and
    // 8.3, 2,000 to 400,000 on 24^3 to 96^3 otherwise the same)
    const uint32_t S = ntiles ? min(4u, max(1u, (gridDim.x + ntiles - 1) / ntiles)) : 1u;
    // this thread's cell of a work item: particles b, b + S, .. < e; the next
    // item's are loaded while this one is summed
    const int64_t N = V.N;
    uint32_t b = 0, e = 0;
    uint4 tile = make_uint4(0u, 0u, 0u, 0u);
    auto cells = [&](uint2 r, const uint4& nt, uint32_t w) {
        b = max(r.x, nt.y) + w % S;
        e = min(r.y, nt.z);
    };
    if (blockIdx.x < ntiles * S) {
        tile = __ldg(&V.ptile[blockIdx.x / S]);
        cells(V.cell_range[(size_t)tile.x * 64 + q], tile, blockIdx.x);
    }
    for (uint32_t w = blockIdx.x; w < ntiles * S; w += gridDim.x) {
        const uint32_t wn = w + gridDim.x;
        const bool more = wn < ntiles * S;
        const uint4 next = more ? __ldg(&V.ptile[wn / S]) : make_uint4(0u, 0u, 0u, 0u);
        float acc[9][4], adj[ADJ ? 9 : 1][3];
#pragma unroll
        for (int o = 0; o < 9; ++o) {
            acc[o][0] = acc[o][1] = acc[o][2] = acc[o][3] = 0.f;
            if (ADJ) adj[o][0] = adj[o][1] = adj[o][2] = 0.f;
        }
        for (uint32_t i = b; i < e; i += S) {
            const float4 q0 = V.q[i], q1 = V.q[N + i], q2 = ADJ ? V.q[2 * N + i] : make_float4(0.f, 0.f, 0.f, 0.f);
            float wx[3], wy[3];
#pragma unroll
            for (int o = 0; o < 3; ++o) {
                wx[o] = ref_cell_weight(q0.x, o);
                wy[o] = ref_cell_weight(q0.y, o);
            }
            const float wz = ref_cell_weight(q0.z, k);
#pragma unroll
            for (int j = 0; j < 3; ++j)
#pragma unroll
                for (int ii = 0; ii < 3; ++ii) {
                    // the reference's product order and threshold
                    float wgt = __fmul_rn(__fmul_rn(wx[ii], wy[j]), wz);
                    wgt = wgt > 1e-10f ? wgt : 0.f;
                    const float wm = __fmul_rn(wgt, q0.w);
                    const int o = 3 * j + ii;
                    acc[o][0] += wm;
                    acc[o][1] += __fmul_rn(wm, q1.x);
                    acc[o][2] += __fmul_rn(wm, q1.y);
                    acc[o][3] += __fmul_rn(wm, q1.z);
                    if (ADJ) {
                        adj[o][0] += wgt * q2.x;
                        adj[o][1] += wgt * q2.y;
                        adj[o][2] += wgt * q2.z;
                    }
                }
        }
        const int lt = (int)tile.x - sc.ct_base;
        const int ox = 4 * (lt % sc.ct[0]), oy = 4 * ((lt / sc.ct[0]) % sc.ct[1]), oz = 4 * (lt / (sc.ct[0] * sc.ct[1]));
        const int l = t & 31, wp = t >> 5;
        const uint2 rn = more ? V.cell_range[(size_t)next.x * 64 + q] : make_uint2(0u, 0u);
        auto flush = [&](float4* grid) {
            auto node = [&](int nx, int ny, int nz) {
                const float4 a4 = slices_node_sum(T4, nx, ny, nz);
                const int gi = ox + nx, gj = oy + ny, gk = oz + nz;
                if ((a4.x != 0.f || a4.y != 0.f || a4.z != 0.f || a4.w != 0.f) && gi < sc.n[0] && gj < sc.n[1] &&
                    gk < sc.n[2])
                    atomicAdd(&grid[node_index(sc, gi, gj, gk)], a4);
            };
            __syncthreads();
            node(l % TN, l / TN, wp);
            if (wp == 0 && l < 24) node(2 + (l & 3), 5, l >> 2);
            __syncthreads();
        };
#pragma unroll
        for (int o = 0; o < 9; ++o)
            T4[k * P2GS_PLANE + o * 64 + q] = make_float4(acc[o][0], acc[o][1], acc[o][2], acc[o][3]);
        flush(V.grid_mp);
        if (ADJ) {
#pragma unroll
            for (int o = 0; o < 9; ++o)
                T4[k * P2GS_PLANE + o * 64 + q] = make_float4(adj[o][0], adj[o][1], adj[o][2], 0.f);
            flush(R.acc);
        }
        tile = next;
        cells(rn, next, wn);
    }
}

// Grid update of the step and of its reverse, over the active node tiles:
// (v, m) to grid_v, (gP, gm) to R.gpm, both accumulators left zero.
__global__ void __launch_bounds__(256) k_ref_grid_adj(View V, RefStep R) {
    if (blockIdx.x == 0 && threadIdx.x < SW_WORDS) V.sort_work[threadIdx.x] = 0u;  // as k_grid
    const SceneDev& sc = V.scenes[0];
    const uint32_t count = V.counters[CNT_TILES];
    const int l = threadIdx.x & 63;
    float acc[3] = {0.f, 0.f, 0.f};
    for (uint32_t w = blockIdx.x * 4 + (threadIdx.x >> 6); w < count; w += gridDim.x * 4) {
        const uint32_t nt = V.tile_list[w];
        if (nt >= (uint32_t)V.total_nt) continue;
        const int64_t idx = ((int64_t)nt << 6) + l;
        const float4 mp = V.grid_mp[idx], g = R.acc[idx];
        float v[3] = {0.f, 0.f, 0.f};
        float4 out = make_float4(0.f, 0.f, 0.f, 0.f);
        if (mp.x > 1e-10f) {
            // material_point_method.h:572-597: p += (m g) dt, v = p / m
            v[0] = __fdiv_rn(__fadd_rn(mp.y, __fmul_rn(__fmul_rn(mp.x, sc.gravity[0]), sc.dt)), mp.x);
            v[1] = __fdiv_rn(__fadd_rn(mp.z, __fmul_rn(__fmul_rn(mp.x, sc.gravity[1]), sc.dt)), mp.x);
            v[2] = __fdiv_rn(__fadd_rn(mp.w, __fmul_rn(__fmul_rn(mp.x, sc.gravity[2]), sc.dt)), mp.x);
            const float im = 1.f / mp.x;
            const float pm0 = v[0] - sc.gravity[0] * sc.dt, pm1 = v[1] - sc.gravity[1] * sc.dt,
                        pm2 = v[2] - sc.gravity[2] * sc.dt;  // P / m
            out = make_float4(g.x * im, g.y * im, g.z * im, -(g.x * pm0 + g.y * pm1 + g.z * pm2) * im);
            acc[0] += g.x;
            acc[1] += g.y;
            acc[2] += g.z;
        }
        V.grid_v[idx] = make_float4(v[0], v[1], v[2], mp.x);
        R.gpm[idx] = out;
        V.grid_mp[idx] = make_float4(0.f, 0.f, 0.f, 0.f);
        R.acc[idx] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    // one atomic per block and component (one per warp on three addresses
    // held the kernel at 14 us)
    __shared__ float s_acc[3][8];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        float s = acc[c] * sc.dt;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xFFFFFFFFu, s, o);
        if ((threadIdx.x & 31) == 0) s_acc[c][threadIdx.x >> 5] = s;
    }
    __syncthreads();
    if (R.ggrav && threadIdx.x < 3) {
        float s = 0.f;
#pragma unroll
        for (int w = 0; w < 8; ++w) s += s_acc[threadIdx.x][w];
        if (s != 0.f) atomicAdd(&R.ggrav[threadIdx.x], s);
    }
}

// One particle's stencil nodes in the reference's loop order (x outer, z
// inner), fn(i, j, k, node index, weight) for weights above the threshold.
template <class Fn>
__device__ __forceinline__ void ref_nodes(const SceneDev& sc, const Stencil& st, const Fn& fn) {
    if (st.b[0] == st.s[0] && st.b[1] == st.s[1] && st.b[2] == st.s[2]) {  // all 27 nodes in the grid
        int X[3], Y[3], Z[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const int gi = st.s[0] + a, gj = st.s[1] + a, gk = st.s[2] + a;
            X[a] = ((gi >> 2) << 6) + (gi & 3);
            Y[a] = (gj >> 2) * (sc.nt[0] << 6) + ((gj & 3) << 2);
            Z[a] = (gk >> 2) * ((sc.nt[0] * sc.nt[1]) << 6) + ((gk & 3) << 4) + (sc.nt_base << 6);
        }
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j)
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const float w = __fmul_rn(__fmul_rn(st.w[0][i], st.w[1][j]), st.w[2][k]);
                    if (w > 1e-10f) fn(i, j, k, (int64_t)(X[i] + Y[j] + Z[k]), w);
                }
        return;
    }
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const int gi = st.b[0] + i;
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const int gj = st.b[1] + j;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const int gk = st.b[2] + k;
                if (gi < 0 || gi >= sc.n[0] || gj < 0 || gj >= sc.n[1] || gk < 0 || gk >= sc.n[2]) continue;
                const float w = __fmul_rn(__fmul_rn(st.w[0][i], st.w[1][j]), st.w[2][k]);
                if (w > 1e-10f) fn(i, j, k, node_index(sc, gi, gj, gk), w);
            }
        }
    }
}

// G2P in the sorted order, into the caller's arrays.
__global__ void __launch_bounds__(128) k_ref_g2p(View V, RefStep R) {
    const SceneDev& sc = V.scenes[0];
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= V.N) return;
    const int64_t p = __float_as_uint(V.q[V.N + i].w);
    if (p >= V.N) {
        atomicOr(&V.counters[CNT_FLAGS], FLAG_TILE_RANGE);
        return;
    }
    uint32_t flags = 0;
    const float x[3] = {R.x[3 * p], R.x[3 * p + 1], R.x[3 * p + 2]};
    Stencil st;
    make_stencil<PHYS_REF>(sc, x, st, flags);
    float nv[3] = {0.f, 0.f, 0.f};
    ref_nodes(sc, st, [&](int, int, int, int64_t idx, float w) {
        const float4 g = __ldg(&V.grid_v[idx]);
        nv[0] = __fadd_rn(nv[0], __fmul_rn(w, g.x));
        nv[1] = __fadd_rn(nv[1], __fmul_rn(w, g.y));
        nv[2] = __fadd_rn(nv[2], __fmul_rn(w, g.z));
    });
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        R.xo[3 * p + c] = __fadd_rn(x[c], __fmul_rn(nv[c], sc.dt));
        R.vo[3 * p + c] = nv[c];
    }
}

// The reverse gather (k_ref_adj_gather's sums) in the sorted order.
__global__ void __launch_bounds__(128) k_ref_gather_sorted(View V, RefStep R) {
    const SceneDev& sc = V.scenes[0];
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= V.N) return;
    const float4 q0 = V.q[i], q1 = V.q[V.N + i], q2 = V.q[2 * V.N + i];
    const int64_t p = __float_as_uint(q1.w);
    if (p >= V.N) {
        atomicOr(&V.counters[CNT_FLAGS], FLAG_TILE_RANGE);
        return;
    }
    uint32_t flags = 0;
    const float xp[3] = {R.x[3 * p], R.x[3 * p + 1], R.x[3 * p + 2]};
    const float vp[3] = {q1.x, q1.y, q1.z}, a[3] = {q2.x, q2.y, q2.z};
    const float mp = q0.w;
    RefStencil r;
    ref_stencil(sc, xp, r, flags);
    float ox[3], ov[3] = {0.f, 0.f, 0.f}, om = 0.f;
#pragma unroll
    for (int c = 0; c < 3; ++c) ox[c] = R.gx[3 * p + c];
    ref_nodes(sc, r.st, [&](int ii, int j, int k, int64_t idx, float w) {
        const float wx = r.st.w[0][ii], wy = r.st.w[1][j], wz = r.st.w[2][k];
        const float4 vi = __ldg(&V.grid_v[idx]);
        const float4 g = __ldg(&R.gpm[idx]);  // (gP, gm)
        const float gPv = g.x * vp[0] + g.y * vp[1] + g.z * vp[2];
        const float s = a[0] * vi.x + a[1] * vi.y + a[2] * vi.z + mp * (g.w + gPv);
        ox[0] += r.dw[0][ii] * wy * wz * s;
        ox[1] += wx * r.dw[1][j] * wz * s;
        ox[2] += wx * wy * r.dw[2][k] * s;
        ov[0] += w * mp * g.x;
        ov[1] += w * mp * g.y;
        ov[2] += w * mp * g.z;
        om += w * (g.w + gPv);
    });
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        R.gx_in[3 * p + c] = ox[c];
        R.gv_in[3 * p + c] = ov[c];
    }
    if (R.gm_in) R.gm_in[p] = om;
}

inline int blocks_for(int64_t n, int block) {
    int64_t g = (n + block - 1) / block;
    return (int)(g < 1 ? 1 : (g > 148 * 64 ? 148 * 64 : g));
}

}  // namespace

cudaError_t launch_ref_adjoint(const View& V, const float* x, const float* v, const float* m, const float* gx,
                               const float* gv, float4* G, float* gx_in, float* gv_in, float* gm_in, float* ggrav,
                               int num_sms, cudaStream_t st) {
    if (V.N == 0) return cudaSuccess;
    k_ref_adj_scatter<<<blocks_for(V.N, 256), 256, 0, st>>>(V, x, gx, gv, G, V.N);
    int nb = (int)std::min<int64_t>(((int64_t)V.total_nt + 3) / 4, (int64_t)num_sms * 8);
    k_ref_adj_grid<<<nb < 1 ? 1 : nb, 256, 0, st>>>(V, G, ggrav);
    k_ref_adj_gather<<<blocks_for(V.N, 256), 256, 0, st>>>(V, x, v, m, gx, gv, G, gx_in, gv_in, gm_in, V.N);
    return cudaGetLastError();
}

cudaError_t launch_ref_step(const View& V, const BinSortBufs& B, const RefStep& R, const PhysFlags& pf,
                            const Tuning& t, int num_sms, cudaStream_t st) {
    if (V.N == 0) return cudaSuccess;
    const bool adj = R.gx != nullptr;
    View K = V;
    K.cnt = B.cnt;
    cudaError_t e = launch_after(false, k_ref_keys, blocks_for(V.N, 256), 256, st, K, R);
    if (e == cudaSuccess) e = bin_sort_step(V, B, num_sms, true, st, &R);
    const int nb = (int)((V.N + 127) / 128);
    if (!adj) {
        if (e == cudaSuccess) e = launch_after(false, k_ref_p2g<false>, num_sms * 4, P2GS_T, st, V, R);
        if (e == cudaSuccess) e = launch_grid(V, pf, t, num_sms, st);
        if (e == cudaSuccess) e = launch_after(false, k_ref_g2p, nb, 128, st, V, R);
    } else {
        const int gb = (int)std::min<int64_t>(((int64_t)V.total_nt + 3) / 4, (int64_t)num_sms * 4);
        if (e == cudaSuccess) e = launch_after(false, k_ref_p2g<true>, num_sms * 3, P2GS_T, st, V, R);
        if (e == cudaSuccess) e = launch_after(false, k_ref_grid_adj, gb < 1 ? 1 : gb, 256, st, V, R);
        if (e == cudaSuccess) e = launch_after(false, k_ref_gather_sorted, nb, 128, st, V, R);
    }
    return e;
}

}  // namespace pgmpm
