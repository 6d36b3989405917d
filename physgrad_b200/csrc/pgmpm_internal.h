// pgmpm_internal.h -- declarations shared by the CUDA translation units of
// libpgmpm.so.  Not installed; the public surface is include/pgmpm.h.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "pgmpm_device.cuh"

namespace pgmpm {

// counters[] layout.  Words [0, CNT_RESET) are cleared every step:
// active node tiles, occupied cell tiles, active node count (u64), the
// work cursors of the tile kernels, and the occupied cell tiles per size
// class (CNT_BUCKETS classes, largest first).  CNT_FLAGS (sticky error
// flags) is cleared only by pgmpm_check_status.
constexpr int CNT_BUCKETS = 8;
enum {
    CNT_TILES = 0,
    CNT_CTILES = 1,
    CNT_ACTIVE = 2,
    CNT_P2G_CURSOR = 4,
    CNT_G2P_CURSOR = 5,
    CNT_BUCKET = 6,
    CNT_RESET = CNT_BUCKET + CNT_BUCKETS,
    CNT_FLAGS = CNT_RESET,
    CNT_STAMP = CNT_RESET + 1,  // sparse grids: step counter; a node tile is active when its flag equals it
    CNT_WORDS = 16
};
static_assert(CNT_STAMP < CNT_WORDS, "counter layout");

// The bin sort's counters (pgmpm_sort.cu): particles per cell and per cell
// tile, and each particle's slot in its cell.  A G2P that another step of the same call follows counts its new keys there
// itself (View::cnt), and that step's sort starts from the counts.
struct SortCounts {
    uint32_t* ccount;      // total_ct * 64 + 1 words (cells + overflow bin)
    uint32_t* tcount;      // total_ct + 1 words
    uint32_t* slot;        // N words
    uint32_t ncells;       // total_ct * 64: keys from here on are out of range
};
// words of the sort's list counters (View::sort_work): occupied cell tiles,
// active node tiles, particles with a key in range, occupied tiles per size
// class.  Zero between steps: the grid update clears them.
enum { SW_CTILES = 0, SW_TILES = 1, SW_VALID = 2, SW_BUCKET = 3, SW_WORDS = 16 };

// Everything a step kernel needs, passed by value.
struct View {
    int64_t N;
    int S, M;
    const SceneDev* scenes;
    const int32_t* scene_tab;  // batched scenes: first scenes of particle / tile blocks (see scene_of)
    const MatDev* mats;
    float4* q;                 // 6 planes of N float4 (state at the start of the step)
    float4* q_out;             // where G2P writes the new state (== q in place; MLS only otherwise)
    float4* pay;               // MLS P2G payload of the state in q (4 planes), read by P2G
    float4* pay_out;           // payload of the state G2P writes (null: G2P does not write one)
    int write_vc;              // MLS G2P stores v and C (planes 3-5); 0 between the steps of one
                               // call, where the next step reads them only through the payload
    const float2* mV;          // (mass, V0)
    const int32_t* mat;        // material id (null when M == 1)
    uint32_t* keys;            // cell key per particle (physical order), input of the next sort
    uint32_t* resort;          // MLS G2P replaying recorded steps: V.keys holds the recorded next
                               // keys; G2P overwrites only those that differ and then sets *resort
                               // (the next step must sort again).  Null: G2P writes every key.
    const uint32_t* skeys;     // sorted keys
    const uint32_t* order;     // sorted position -> physical particle
    float4* grid_mp;           // (m, p) accumulator
    float4* grid_v;            // (v, m) after the grid update
    float4* grid_vpre;         // optional: (v before walls, m), recorded for the adjoint
    uint32_t* tile_flags;      // node tile active flags (per global node tile)
    uint32_t* tile_list;       // active node tiles
    uint32_t* ctile_list;      // occupied cell tiles (global cell tile ids)
    const uint4* ptile;        // bin sort: the occupied cell tiles, largest first, as (tile, first
                               // sorted position, end, scene); null (radix sort): use ctile_list
    uint2* ctile_range;        // per global cell tile: [begin, end) in sorted order
    const uint2* cell_range;   // per global cell: [begin, end) in sorted order (null: search skeys)
    uint32_t* counters;        // see CNT_*
    uint32_t* sort_work;       // see SW_* (null without the bin sort)
    bool early;                // launches of this step may be early (see launch_after),
    bool early_first;          // its first one too: a step kernel precedes it on the stream
    SortCounts cnt;            // counters a G2P counts its new keys into (ccount null: it does not)
    int total_ct, total_nt;
    SparseTiles sp;            // sparse grid (sp.cap == 0: dense; tile ids are then slots)
};

// Scene of a particle, cell tile or node tile of a batched solver.  scene_tab
// holds the scene of the first particle of every SCENE_BLOCK_P particles, then
// of the first of every SCENE_BLOCK_T cell tiles and node tiles, so a lookup
// is one table load and a walk over the scenes that begin inside the block
// (usually none) where a search over the scene table would be log2(S)
// dependent loads per particle (64 scenes, 3.9 M particles, 10 steps between
// an upload and a download: 7263 -> 7187 us; forward + adjoint of 12 scenes,
// 24 steps: 4359 -> 4336 us).
constexpr int SCENE_BLOCK_P = 128;
constexpr int SCENE_BLOCK_T = 64;
inline __host__ __device__ int64_t scene_tab_ct(int64_t N) { return (N + SCENE_BLOCK_P - 1) / SCENE_BLOCK_P; }
inline __host__ __device__ int64_t scene_tab_nt(int64_t N, int total_ct) {
    return scene_tab_ct(N) + ((int64_t)total_ct + SCENE_BLOCK_T - 1) / SCENE_BLOCK_T;
}
inline __host__ __device__ int64_t scene_tab_size(int64_t N, int total_ct, int total_nt) {
    return scene_tab_nt(N, total_ct) + ((int64_t)total_nt + SCENE_BLOCK_T - 1) / SCENE_BLOCK_T;
}
__device__ __forceinline__ int scene_of_particle(const View& V, int64_t p) {
    if (V.S == 1) return 0;
    int s = __ldg(&V.scene_tab[p / SCENE_BLOCK_P]);
    while (s + 1 < V.S && __ldg(&V.scenes[s + 1].p_begin) <= p) ++s;
    return s;
}
__device__ __forceinline__ int scene_of_cell_tile(const View& V, int ct) {
    if (V.S == 1) return 0;
    int s = __ldg(&V.scene_tab[scene_tab_ct(V.N) + ct / SCENE_BLOCK_T]);
    while (s + 1 < V.S && __ldg(&V.scenes[s + 1].ct_base) <= ct) ++s;
    return s;
}
__device__ __forceinline__ int scene_of_node_tile(const View& V, int nt) {
    if (V.S == 1) return 0;
    int s = __ldg(&V.scene_tab[scene_tab_nt(V.N, V.total_ct) + nt / SCENE_BLOCK_T]);
    while (s + 1 < V.S && __ldg(&V.scenes[s + 1].nt_base) <= nt) ++s;
    return s;
}

// One occupied cell tile of the step: its index, its particles' range in the
// sorted order, its scene.
struct TileWork {
    uint32_t ct;
    uint2 rg;
    int s;
};
__device__ __forceinline__ TileWork tile_work(const View& V, uint32_t w) {
    if (V.ptile) {
        const uint4 t = __ldg(&V.ptile[w]);
        return {t.x, make_uint2(t.y, t.z), (int)t.w};
    }
    const uint32_t ct = V.ctile_list[w];
    return {ct, V.ctile_range[ct], scene_of_cell_tile(V, (int)ct)};
}

// Counts key k into the sort's counters: adds each run of equal keys among
// the active lanes with one atomic.  Returns the run's first slot in its
// first lane (in flight until used); run_slot() gives each lane its own.
struct KeyRun {
    uint32_t mask;  // lanes that count together
    int start;      // first lane of this lane's run
    uint32_t base;  // the run's first slot, in lane `start`
};
__device__ __forceinline__ KeyRun count_key(const SortCounts& c, uint32_t k) {
    const uint32_t m = __activemask();
    const int lane = threadIdx.x & 31;
    const uint32_t upto = lane == 31 ? 0xFFFFFFFFu : ((2u << lane) - 1u);  // lanes <= this one
    const uint32_t prev = __shfl_up_sync(m, k, 1);
    const bool first = lane == 0 || !((m >> (lane - 1)) & 1u);
    const bool head = first || prev != k;
    const bool thead = first || (prev ^ k) >> 6;
    // a run ends before the next head or the next inactive lane
    auto end_of = [&](uint32_t heads) {
        const uint32_t stop = (heads | ~m) & ~upto;
        return stop ? __ffs(stop) - 1 : 32;
    };
    const uint32_t heads = __ballot_sync(m, head), theads = __ballot_sync(m, thead);
    KeyRun r;
    r.mask = m;
    r.start = 31 - __clz(heads & upto);
    r.base = head ? atomicAdd(&c.ccount[k], (uint32_t)(end_of(heads) - lane)) : 0u;
    if (thead) atomicAdd(&c.tcount[k >> 6], (uint32_t)(end_of(theads) - lane));
    return r;
}
__device__ __forceinline__ uint32_t run_slot(const KeyRun& r) {
    return __shfl_sync(r.mask, r.base, r.start) + (uint32_t)((threadIdx.x & 31) - r.start);
}

// Launches of a step's kernels.  They are a few us each and depend on one
// another; an early launch (programmatic stream serialization) sets the grid
// up while the kernel before it on the stream drains, and its threads wait in
// step_wait() for that kernel's end.  Early only right after a kernel (not
// after a copy, a memset, an event, a graph or a conditional node), and only
// kernels that begin with step_wait(): since each waits for the one before (or is
// launched the plain way), order holds along the whole chain.  32,768 particles
// 1374 -> 1306 us for 50 steps; at 2 M the same time.  The kernels do not signal
// their successors before their end: blocks that wait on the SM keep the running
// kernel's out (262,144 particles with gradients 6733 -> 7024 us).  G2P is
// launched the plain way: its node reads want the read-only path (plain loads:
// 96 -> 108 us at 2 M), and the early launch gave it nothing on top.  The status
// is the launch's own, not an error that something else left in the thread.
template <class... P, class... A>
inline cudaError_t launch_after(bool early, void (*kernel)(P...), int grid, int block, cudaStream_t st, A... a) {
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3((unsigned)grid);
    c.blockDim = dim3((unsigned)block);
    c.stream = st;
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    c.attrs = &at;
    c.numAttrs = early ? 1 : 0;
    return cudaLaunchKernelEx(&c, kernel, static_cast<P>(a)...);
}

// P2G variants: 0 = (cell, z-slice) register accumulation with a staged
// payload, 1 = per-particle shared-memory atomics over fixed chunks,
// 2 = one thread per cell, 108 register accumulators, no staging,
// 3 = variant 2 with a cell's accumulators split over two lanes (MLS
// forward; the REF physics and the adjoint scatter run variant 2).
// G2P variant 2 = direct gather in physical particle order (default).
// G2P variants: 0 = node tile staged in shared memory, 1 = direct gather.
struct Tuning {
    int p2g_block = 192;   // variant 0 uses exactly 192 threads (64 cells x 3 z-slices)
    int ppt = 1024;        // variant 1: particles per chunk; variant 0: sub-chunk staged at once is fixed
    int g2p_block = 128;   // 64..512 swept: 64 and 128 equal, 192..512 up to 2.5% slower
    int grid_block = 256;
    int p2g_variant = 2;
    int g2p_variant = 2;
    int tile_blocks_per_sm = 3;  // persistent P2G tile kernel: blocks per SM
    int g2p_tiles_per_sm = 2;    // persistent G2P tile kernel: blocks per SM (256 threads)
    int cell_blocks_per_sm = 6;  // persistent P2G thread-per-cell kernel (variant 2): blocks per SM
    int pair_blocks_per_sm = 5;  // persistent P2G two-threads-per-cell kernel (variant 3): blocks per SM
    int step_sort = 0;           // per-step sort: 0 = bin sort (counting sorts by tile, then cell), 1 = radix sort
    int g2p2g_blocks_per_sm = 4; // fused kernel (P2G variant 5): 4 (255 registers) or 6 (168, some spilled)
};
// P2G variant 5 = variant 4's P2G, fused with the previous step's G2P when
// steps follow one another (launch_g2p2g).

// What one recorded step launches.  MLS with the fused G2P -> P2G kernel
// (P2G variant 5) chains steps: a step's G2P2G does the next step's P2G.
enum StepKind {
    STEP_SPLIT = 0,    // sort, P2G, grid update, G2P (which writes the next payload)
    STEP_FUSED_FIRST,  // sort, P2G, grid update, G2P2G
    STEP_FUSED,        // sort, grid update, G2P2G (P2G done by the previous step's G2P2G)
    STEP_FUSED_LAST,   // sort, grid update, G2P (nothing left pending in grid_mp)
    STEP_KINDS
};

// pgmpm_sort.cu
constexpr int RADIX_TILE = 2048;  // keys per block of the sort kernels
constexpr int RADIX_MAX_DIGITS = 256;
// u32 words of histogram scratch the sort needs for n pairs
constexpr int64_t radix_scratch_words_for(int64_t n) {
    return ((n + RADIX_TILE - 1) / RADIX_TILE) * RADIX_MAX_DIGITS + RADIX_MAX_DIGITS;
}
int64_t radix_sort_scratch_words(int64_t n);
int radix_passes(int key_bits);
cudaError_t radix_sort_pairs(const uint32_t* kin, const uint32_t* vin, uint32_t* ka, uint32_t* va, uint32_t* kb,
                             uint32_t* vb, uint32_t* scratch, int64_t n, int key_bits, int* which,
                             cudaStream_t st);

// One REF_COMPAT step on the caller's arrays (bin sort): the forward (gx null:
// new positions and velocities to xo, vo, which may be x and v) or the reverse
// of the step from x, v, m (gx_in, gv_in, gm_in (may be null), ggrav added to).
struct RefStep {
    const float *x, *v, *m;  // [N][3], [N][3], [N]
    const float* gravity;    // device [3], copied into the scene; null: the scene's
    float* keep_m;           // copy of m (or m itself)
    float *xo, *vo;
    const float *gx, *gv;
    float *gx_in, *gv_in, *gm_in, *ggrav;
    float4* acc;             // per node, zero between calls
    float4* gpm;             // per node
};

// Per-step bin sort (pgmpm_sort.cu): keys_in (physical order) -> out_k /
// out_v sorted by key, plus the occupied cell tiles with their ranges
// (largest first), every cell's [begin, end) in the sorted order of the
// occupied tiles, and the active node tiles and their flags (View fields).
// The counters of cnt must be zero on entry, or (counted) hold the counts of
// keys_in, and are left zero; V.sort_work must be zero, and the step's grid
// update clears it again.
struct BinSortBufs {
    const uint32_t* keys_in;
    SortCounts cnt;
    uint32_t *out_k, *out_v;  // N words each
    uint2* cell_range;     // total_ct * 64
    uint4* ptile;          // total_ct: see View::ptile
    uint4* tile_info;      // total_ct: (tile, begin, end, class << 28 | rank) in order of discovery (scratch)
    uint32_t* gsum;        // bin_sort_groups(total_ct) words (scratch)
};
int64_t bin_sort_groups(int64_t total_ct);
// rec: write the particles' records to the state planes instead of out_k, out_v
cudaError_t bin_sort_step(const View& V, const BinSortBufs& B, int num_sms, bool counted, cudaStream_t st,
                          const RefStep* rec = nullptr);

// pgmpm_kernels.cu
struct PhysFlags {
    int physics;     // PHYS_MLS / PHYS_REF (same for every scene)
    bool multi_mat;  // per-particle material ids
    bool has_fluid;  // some material uses the EOS model
    bool has_plastic;  // some material is ELASTOPLASTIC (von Mises)
};
// x: the caller's positions, upload order; writes V.keys in that order
cudaError_t launch_keys(const View& V, const float* x, const PhysFlags& pf, cudaStream_t st);
cudaError_t launch_payload(const View& V, const PhysFlags& pf, cudaStream_t st);
cudaError_t launch_mark(const View& V, cudaStream_t st);
cudaError_t launch_p2g(const View& V, const PhysFlags& pf, const Tuning& t, int num_sms, cudaStream_t st);
cudaError_t launch_grid(const View& V, const PhysFlags& pf, const Tuning& t, int num_sms, cudaStream_t st);
cudaError_t launch_g2p(const View& V, const PhysFlags& pf, const Tuning& t, int num_sms, cudaStream_t st);
// Fused G2P of this step and P2G of the next (MLS with the bin sort's cell
// table): writes the new state and keys and accumulates the next step's
// (m, p) into V.grid_mp; takes work from the G2P cursor.
cudaError_t launch_g2p2g(const View& V, const PhysFlags& pf, const Tuning& t, int num_sms, cudaStream_t st);
cudaError_t launch_pack(const View& V, const float* x, const float* v, const float* C, const float* F,
                        const float* m, const float* V0, const int32_t* mat, const uint32_t* order,
                        const uint32_t* skeys, uint32_t* user_of_phys, uint32_t* phys_of_user, float2* mV_out,
                        int32_t* mat_out, cudaStream_t st);
// phys_of_user: upload index -> physical slot (written by launch_pack)
cudaError_t launch_unpack(const View& V, const uint32_t* phys_of_user, float* x, float* v, float* C, float* F,
                          cudaStream_t st);
// ORs the error flags of `slots` counter blocks (stride CNT_WORDS) into
// live[CNT_FLAGS] and clears them.
cudaError_t launch_merge_flags(uint32_t* slots_counters, int slots, uint32_t* live, cudaStream_t st);
cudaError_t launch_grid_download(const View& V, int scene, const SceneDev& sc, float* mass, float* vel,
                                 cudaStream_t st);

// Reverse pass of one MLS step (pgmpm_adjoint.cu, and the scatter in
// pgmpm_kernels.cu).  V describes the step as it ran (V.q = state before the
// step, order / tiles / grid_v / grid_vpre of the step); V.grid_mp is the
// scatter target for dL/dv_i.
struct AdjView {
    // adjoint of the particle state after the step, overwritten with the
    // adjoint of the state before it (physical order, same plane packing)
    float4* g;                 // 6 planes
    const float4* q_next;      // state after the step (C' for the F update and the fluid reset)
    float4* pay;               // the scatter's payload (4 planes of N float4)
    bool pay_ready;            // pay holds this step's already
    const float4* q_prev;      // state before the step before: the gather forms that step's payload (or null)
    float4* grid_gv;           // (0, dL/dv_i) scatter target, zeroed by the grid adjoint
    float4* grid_gpm;          // (dL/dp_i, dL/dm_i) per node
    float* gE;                 // [M] dL/dE accumulators
};
// launch_adj_scatter runs from A.pay (P2G variants 4 and 5 with the bin sort,
// where there was memory for it)
inline bool adj_scatter_from_payload(const View& V, const AdjView& A, const Tuning& t) {
    return t.p2g_variant >= 4 && V.cell_range && A.pay;
}
cudaError_t launch_adj_scatter(const View& V, const AdjView& A, const PhysFlags& pf, const Tuning& t, int num_sms,
                               cudaStream_t st);
cudaError_t launch_adj_grid(const View& V, const AdjView& A, const Tuning& t, int num_sms, cudaStream_t st);
cudaError_t launch_adj_gather(const View& V, const AdjView& A, const PhysFlags& pf, const Tuning& t,
                              cudaStream_t st);
cudaError_t launch_state_to_planes(const float* x, const float* v, const float* C, const float* F,
                                   const uint32_t* user_of_phys, float4* g, int64_t N, cudaStream_t st);
// reverse of one REF_COMPAT step (pgmpm_ref_adjoint.cu); particle arrays in
// the caller's order, G: one float4 per grid node, zeroed by the caller
cudaError_t launch_ref_adjoint(const View& V, const float* x, const float* v, const float* m, const float* gx,
                               const float* gv, float4* G, float* gx_in, float* gv_in, float* gm_in, float* ggrav,
                               int num_sms, cudaStream_t st);
cudaError_t launch_ref_step(const View& V, const BinSortBufs& B, const RefStep& R, const PhysFlags& pf,
                            const Tuning& t, int num_sms, cudaStream_t st);
cudaError_t launch_planes_to_state(const float4* g, const uint32_t* phys_of_user, float* x, float* v, float* C,
                                   float* F, int64_t N, cudaStream_t st);

}  // namespace pgmpm
