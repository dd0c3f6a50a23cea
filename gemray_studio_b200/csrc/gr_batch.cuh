// gr_batch.cuh -- batched launches: many scenes (each with its own planes, material,
// environment and film) in one grid.  Included by gr_batch.cu only.
#pragma once

#include "gr_transport.cuh"

namespace grd {

// A segment is one scene's run of whole pixels for one sample
// range; every block of the trace kernel (every warp of the fold kernel) belongs to
// exactly one segment, found by binary search over the segments' first block (warp).
// The scene's constants are copied into shared memory, so per-tuple arithmetic is
// that of the single-scene kernel and results are bit-identical to rendering each
// scene alone.
struct SceneSlot {
    SceneConst S;
    SceneBuffers B;
};

struct BatchSegment {
    LaunchRange R;         // pixels / samples of this segment
    float *xyz;            // its per-tuple XYZ (3 f32 per tuple)
    float *film;           // the scene's film (W*H*3 f32), folded into (fold_pixel)
    float *comp;           // continue mode with Kahan: the film's compensation terms
    uint64_t block_begin;  // first trace block of the segment
    uint64_t warp_begin;   // first fold warp of the segment
    uint32_t scene;        // index into the SceneSlot table
    uint32_t kahan;
    uint32_t cont;         // fold_pixel continue mode
    uint32_t park_cap;     // park slots of this segment (paths alive after the stage cap)
    uint32_t stage_cap;    // stage-1 bounce cap: the scene's chosen one (StageCapTune)
    uint64_t park_off;     // first park slot of this segment in the launch's park buffer
    uint64_t park_block_begin;  // first continuation block of the segment
};

// KEY 0: trace blocks, 1: fold warps, 2: continuation blocks.
template <int KEY>
__device__ __forceinline__ uint32_t find_segment(const BatchSegment *__restrict__ segs, uint32_t n, uint64_t key) {
    uint32_t lo = 0, hi = n;  // last segment whose begin <= key
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        const uint64_t b = KEY == 1 ? segs[mid].warp_begin : (KEY == 2 ? segs[mid].park_block_begin : segs[mid].block_begin);
        if (b <= key) lo = mid;
        else hi = mid;
    }
    return lo;
}

__device__ __forceinline__ void load_slot(SceneSlot &dst_slot, const SceneSlot *__restrict__ src_slot) {
    const uint32_t *src = reinterpret_cast<const uint32_t *>(src_slot);
    uint32_t *dst = reinterpret_cast<uint32_t *>(&dst_slot);
    for (uint32_t i = threadIdx.x; i < sizeof(SceneSlot) / 4; i += blockDim.x) dst[i] = src[i];
}

// A batched launch in the plain kernel's form (gr_transport.cuh): `lanes` tuples of one segment
// per warp, run to their ends.
template <bool EXTRAS, int K = K_ANY>
__global__ void __launch_bounds__(TRACE_THREADS, GR_TRACE_MIN_BLOCKS)
    k_trace_batch_plain(const SceneSlot *__restrict__ slots, const BatchSegment *__restrict__ segs, uint32_t n_segs,
                        uint32_t lanes) {
    __shared__ SceneSlot s_slot;
    __shared__ uint32_t s_seg;
    extern __shared__ float4 s_planes[];
    if (threadIdx.x == 0) s_seg = find_segment<0>(segs, n_segs, blockIdx.x);
    __syncthreads();
    const BatchSegment &G = segs[s_seg];
    load_slot(s_slot, slots + G.scene);
    __syncthreads();
    const SceneConst &S = s_slot.S;
    const SceneBuffers &B = s_slot.B;
    const Planes PL = stage_scene_planes<EXTRAS, K>(s_planes, S, B);
    const LaunchRange R = G.R;
    const uint64_t t = plain_tuple(blockIdx.x - G.block_begin, lanes, R.n_tuples);
    if (t >= R.n_tuples) return;
    uint32_t pixel, sample;
    tuple_coords(R, t, pixel, sample);
    Path P;
    path_init<K>(P, S, pixel, sample, (uint32_t)t);
    NoCounters nc;
    store_sample(G.xyz, P, trace_path<NoCounters, false, EXTRAS, K>(P, S, B, PL, nc));
}

// Stage 1 of a batched launch (the pooled scheme of the single-scene kernels): a block runs
// its pool over one segment's run of `chunk` tuples; once they are all started, paths past
// the segment's stage cap are parked in its park region (`park`, slot counters `counts` per
// segment of the launch) for k_trace_batch_cont.
// EXTRAS: the variant for launches holding a scene with frosted facets, scattering or
// a biaxial material.  K: the scene class every segment of the launch belongs to
// (gr_trace.cuh K_*; K_ANY: checked at run time), MB: resident blocks per SM.
template <bool EXTRAS, int K = K_ANY, int MB = GR_TRACE_MIN_BLOCKS>
__global__ void __launch_bounds__(pool_threads<EXTRAS, K>(), pool_blocks(MB, pool_threads<EXTRAS, K>()))
    k_trace_batch(const SceneSlot *__restrict__ slots, const BatchSegment *__restrict__ segs, uint32_t n_segs,
                  uint32_t chunk, Path *__restrict__ park, unsigned int *__restrict__ counts) {
    __shared__ SceneSlot s_slot;
    __shared__ uint32_t s_seg;
    extern __shared__ float4 s_planes[];
    if (threadIdx.x == 0) s_seg = find_segment<0>(segs, n_segs, blockIdx.x);
    __syncthreads();
    const BatchSegment &G = segs[s_seg];
    load_slot(s_slot, slots + G.scene);
    __syncthreads();
    const SceneConst &S = s_slot.S;
    const SceneBuffers &B = s_slot.B;
    Planes PL = stage_scene_planes<EXTRAS, K>(s_planes, S, B);
    stage_camera_table(PL, s_planes + planes_smem_bytes(S.n_planes) / sizeof(float4), ld3(S.cam_o));
    const LaunchRange R = G.R;
    const uint64_t first = (uint64_t)(blockIdx.x - G.block_begin) * chunk;
    float *xyz = G.xyz;
    __shared__ HeroOrder H;
    if (R.spp >= HERO_MIN_SPP) hero_order(H, R);
    Path P;
    run_pool<pool_threads<EXTRAS, K>(), EXTRAS, K, true>(
        P, S, B, PL, PoolRange{first, min(first + chunk, R.n_tuples)}, G.stage_cap,
        ParkOut{park + G.park_off, G.park_cap, counts + s_seg},
        [&](Path &q, uint64_t t) {
            uint32_t px, s;
            hero_coords(R, H, t, px, s);
            path_init<K>(q, S, R.first_pixel + px, R.sample_offset + s, px * R.spp + s);
        },
        [&](const Path &q) { store_sample(xyz, q, path_finish<1, false, K, EXTRAS>(q, S, B)); });
}

// Stage 2: each block resumes up to a block's worth of one segment's parked paths (its scene
// in shared memory, as in stage 1) and runs them to their end.
template <bool EXTRAS, int K = K_ANY, int MB = GR_TRACE_MIN_BLOCKS>
__global__ void __launch_bounds__(pool_threads<EXTRAS, K>(), pool_blocks(MB, pool_threads<EXTRAS, K>()))
    k_trace_batch_cont(const SceneSlot *__restrict__ slots, const BatchSegment *__restrict__ segs, uint32_t n_segs,
                       const Path *__restrict__ park, const unsigned int *__restrict__ counts) {
    __shared__ SceneSlot s_slot;
    __shared__ uint32_t s_seg;
    extern __shared__ float4 s_planes[];
    if (threadIdx.x == 0) s_seg = find_segment<2>(segs, n_segs, blockIdx.x);
    __syncthreads();
    const BatchSegment &G = segs[s_seg];
    const uint32_t n = min((uint32_t)counts[s_seg], G.park_cap);
    const uint64_t j0 = (uint64_t)(blockIdx.x - G.park_block_begin) * blockDim.x;
    if (j0 >= n) return;  // block-uniform: no thread of this block reaches a barrier
    load_slot(s_slot, slots + G.scene);
    __syncthreads();
    const SceneConst &S = s_slot.S;
    const SceneBuffers &B = s_slot.B;
    const Planes PL = stage_scene_planes<EXTRAS, K>(s_planes, S, B);
    const Path *from = park + G.park_off;
    float *xyz = G.xyz;
    Path P;
    run_pool<pool_threads<EXTRAS, K>(), EXTRAS, K, false>(
        P, S, B, PL, PoolRange{j0, min(j0 + blockDim.x, (uint64_t)n)}, 0xFFFFFFFFu, ParkOut{nullptr, 0, nullptr},
        [&](Path &q, uint64_t i) { copy_record<record_rows<EXTRAS, K>()>(q, from[i]); },
        [&](const Path &q) { store_sample(xyz, q, path_finish<1, false, K, EXTRAS>(q, S, B)); });
}

// The trace grids of one batched launch: its segments, scratch and grid sizes (gr_batch.cu).
// lanes: the plain form with that many tuples per warp; 0: the pooled form's two grids.
struct BatchLaunch {
    const SceneSlot *slots;
    const BatchSegment *segs;
    uint32_t n_segs, lanes, chunk, max_planes;
    uint64_t blocks, park_blocks;
    Path *park;
    unsigned int *counts;
};

// They, for scene class K with MB blocks per SM in the pooled form.
template <bool EXTRAS, int K, int MB>
void launch_batch_grids(const BatchLaunch &L, cudaStream_t s) {
    const size_t smem = planes_smem_bytes(L.max_planes);
    if (L.lanes) {
        k_trace_batch_plain<EXTRAS, K><<<(unsigned)L.blocks, TRACE_THREADS, smem, s>>>(L.slots, L.segs, L.n_segs, L.lanes);
        return;
    }
    constexpr int T = pool_threads<EXTRAS, K>();
    k_trace_batch<EXTRAS, K, MB><<<(unsigned)L.blocks, T, smem + camera_smem_bytes(L.max_planes), s>>>(
        L.slots, L.segs, L.n_segs, L.chunk, L.park, L.counts);
    k_trace_batch_cont<EXTRAS, K, MB><<<(unsigned)L.park_blocks, T, smem, s>>>(L.slots, L.segs, L.n_segs, L.park, L.counts);
}

}  // namespace grd
