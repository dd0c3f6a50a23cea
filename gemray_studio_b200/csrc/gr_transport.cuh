// gr_transport.cuh -- the single-scene transport kernels (sm_100a): the plain kernel
// (one thread per tuple) and the pooled ones (k_trace_pool, k_trace_resume; the scheme is in
// gr_stage.cuh), templates over the scene class K (gr_trace.cuh) so that each class is compiled
// with only the code it runs.  Instantiated by gr_host.cu (the run-time class, counters, FP64
// re-solve, extension materials) and by gr_single_*.cu (the specialised classes).
#pragma once

#include "gr_stage.cuh"

namespace grd {

// The thread's tuple in block `block` of a plain launch of `lanes` tuples per warp; `none` for
// the other lanes.
__device__ __forceinline__ uint64_t plain_tuple(uint64_t block, uint32_t lanes, uint64_t none) {
    const uint32_t lane = threadIdx.x & 31u;
    return lane < lanes ? (block * (blockDim.x / 32u) + threadIdx.x / 32u) * lanes + lane : none;
}

// Plain kernel: one thread traces one tuple start to finish, `lanes` tuples per warp -- the reference
// kernel's launch shape (one invocation per (pixel, sample), spectral_transport.wgsl:
// 672-691).  The Counters variant tallies events for the FLOP model; RESOLVE is the
// GR_FLAG_FP64_RESOLVE variant (FP64 re-solve of ambiguous exits and TIR decisions);
// EXTRAS the variant for scenes with frosted facets, volume scattering or a biaxial
// material.
template <class CT, bool RESOLVE = false, bool EXTRAS = false, int K = K_ANY, int MB = GR_TRACE_MIN_BLOCKS>
__global__ void __launch_bounds__(TRACE_THREADS, MB) k_trace_plain(SceneConst S, SceneBuffers B, LaunchRange R,
                                                               float *__restrict__ xyz,
                                                               unsigned long long *__restrict__ tallies,
                                                               uint32_t lanes = 32) {
    extern __shared__ float4 s_planes[];
    const Planes PL = stage_scene_planes<EXTRAS, K>(s_planes, S, B);
    const uint64_t t = plain_tuple(blockIdx.x, lanes, R.n_tuples);
    CT ct;
    if constexpr (sizeof(CT) == sizeof(Counters)) {
        for (int i = 0; i < C_COUNT; ++i) ((Counters &)ct).c[i] = 0;
    }
    if (t < R.n_tuples) {
        uint32_t pixel, sample;
        tuple_coords(R, t, pixel, sample);
        Path P;
        path_init<K>(P, S, pixel, sample, (uint32_t)t);
        tally(ct, C_PATHS);
        V3 c = trace_path<CT, RESOLVE, EXTRAS, K>(P, S, B, PL, ct);
        xyz[3 * t + 0] = c.x;
        xyz[3 * t + 1] = c.y;
        xyz[3 * t + 2] = c.z;
    }
    if constexpr (sizeof(CT) == sizeof(Counters)) {
        const uint32_t lane = threadIdx.x & 31u;
        for (int i = 0; i < C_COUNT; ++i) {
            unsigned long long v = ((Counters &)ct).c[i];
            for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
            if (lane == 0 && v) atomicAdd(tallies + i, v);
        }
    }
}

// Paths per warp of a plain launch.  A launch that leaves the chip idle waits for its longest
// path, and a warp runs the branches and channels of all its paths in turn: fewer paths per
// warp shorten that chain while each of the 4 x 148 schedulers has few warps.  Measured on
// the 73-plane brilliant, studio, depth 32 (us at 32 / 16 / 8 / 4 paths per warp): 4,608
// tuples 339 / 296 / 278 / 253 clear, 211 / 185 / 169 / 155 birefringent, 725 / 717 / 647 /
// 643 biaxial; 16,384 tuples 348 / 309 / 295 / 317, 259 / 244 / 257 / 282, 771 / 738 / 751 /
// 902; 36,864 tuples 405 / 348 / 351 / 412, 263 / 304 / 325 / 445, 780 / 863 / 1023 / 1280.
inline uint32_t plain_lanes(uint64_t n_tuples, bool clear) {
    const uint64_t per_lane = 4 * 4 * 148;  // four warps on every scheduler of the B200's 148 SMs
    if (n_tuples <= 4 * per_lane) return 4;
    if (clear) return n_tuples <= 8 * per_lane ? 8 : (n_tuples <= 16 * per_lane ? 16 : 32);
    return n_tuples <= 8 * per_lane ? 16 : 32;
}
inline unsigned plain_blocks(uint64_t n_tuples, uint32_t lanes) {
    const uint64_t per = (uint64_t)lanes * (TRACE_THREADS / 32);
    return (unsigned)((n_tuples + per - 1) / per);
}

// Batched launches and Stokes films of fewer tuples run in the plain form: the pool's blocks of
// 256 or 512 threads leave most of the chip idle there and wait at their barriers for the
// longest scan of the block.  Measured, us of a call, plain / pool.  Batches: quartz cube 2,048
// tuples 92 / 200, 131,072 394 / 420, 262,144 596 / 544; clear brilliant 16,384 279 / 438,
// 131,072 454 / 529, 262,144 684 / 636; emerald 131,072 682 / 769, 262,144 967 / 860; frosted
// biaxial 16,384 852 / 1002, 32,768 977 / 972, 65,536 1285 / 1066.  Stokes films (no scene
// class): cube 2,048 155 / 258, 131,072 370 / 366; brilliant 65,536 472 / 740, 262,144 835 /
// 1058; emerald 131,072 624 / 750, 262,144 878 / 885, 393,216 1523 / 1396; frosted biaxial
// 16,384 964 / 1337, 65,536 1386 / 1368, 131,072 1970 / 1562.
inline uint64_t plain_tuples(bool extras) { return extras ? 1u << 16 : 1u << 18; }

// Pooled kernels (the scheme and run_pool are in gr_stage.cuh), three launches per trace:
// k_trace_pool over the launch's tuples, then k_trace_resume over the paths it parked past
// the first cap and again over those parked past the second, to their ends.
// MB: resident blocks per SM the register allocation targets, in blocks of 128 threads (the
// schedule tuner's dimension).  work: the launch's zeroed tuple counter.
template <bool EXTRAS, int K = K_ANY, int MB = GR_TRACE_MIN_BLOCKS>
__global__ void __launch_bounds__(pool_threads<EXTRAS, K>(), pool_blocks(MB, pool_threads<EXTRAS, K>()))
    k_trace_pool(SceneConst S, SceneBuffers B, LaunchRange R, float *__restrict__ xyz, unsigned long long *work,
                 ParkOut out, uint32_t bounce_cap) {
    extern __shared__ float4 s_planes[];
    Planes PL = stage_scene_planes<EXTRAS, K>(s_planes, S, B);
    stage_camera_table(PL, s_planes + planes_smem_bytes(S.n_planes) / sizeof(float4), ld3(S.cam_o));
    __shared__ HeroOrder H;
    if (R.spp >= HERO_MIN_SPP) hero_order(H, R);
    Path P;
    run_pool<pool_threads<EXTRAS, K>(), EXTRAS, K, true>(
        P, S, B, PL, PoolQueue{work, R.n_tuples}, bounce_cap, out,
        [&](Path &q, uint64_t t) {
            uint32_t px, s;
            hero_coords(R, H, t, px, s);
            path_init<K>(q, S, R.first_pixel + px, R.sample_offset + s, px * R.spp + s);
        },
        [&](const Path &q) { store_sample(xyz, q, path_finish<1, false, K, EXTRAS>(q, S, B)); });
}

// Parked paths [0, min(*count_in, cap_in)), up to `bounce_cap`, survivors parked in `out`
// (out.cap 0: to the end).
template <bool EXTRAS, int K = K_ANY, int MB = GR_TRACE_MIN_BLOCKS>
__global__ void __launch_bounds__(pool_threads<EXTRAS, K>(), pool_blocks(MB, pool_threads<EXTRAS, K>()))
    k_trace_resume(SceneConst S, SceneBuffers B, const Path *__restrict__ park_in, uint32_t cap_in,
                   const unsigned int *__restrict__ count_in, uint32_t bounce_cap, unsigned long long *work, ParkOut out,
                   float *__restrict__ xyz) {
    const uint32_t n = min((uint32_t)*count_in, cap_in);
    if ((uint64_t)blockIdx.x * blockDim.x >= n) return;  // more blocks than parked paths fill
    extern __shared__ float4 s_planes[];
    const Planes PL = stage_scene_planes<EXTRAS, K>(s_planes, S, B);
    Path P;
    run_pool<pool_threads<EXTRAS, K>(), EXTRAS, K, false>(
        P, S, B, PL, PoolQueue{work, n}, bounce_cap, out,
        [&](Path &q, uint64_t i) { copy_record<record_rows<EXTRAS, K>()>(q, park_in[i]); },
        [&](const Path &q) { store_sample(xyz, q, path_finish<1, false, K, EXTRAS>(q, S, B)); });
}

// The three launches of a pooled trace (`work`: three zeroed counters, one per stage; `grid`
// blocks at most, as many as stay resident).
struct PoolLaunch {
    Path *park1, *park2;
    uint32_t cap1, cap2;  // slots
    unsigned int *counts;
    unsigned long long *work;
    uint32_t cap_first, cap_second;
    int sm_count;
    bool alone;  // the first launch only, nothing parked
};
template <bool EXTRAS, int K, int MB>
void launch_pool(const SceneConst &S, const SceneBuffers &B, const LaunchRange &R, float *xyz, cudaStream_t stream,
                 const PoolLaunch &L) {
    constexpr int T = pool_threads<EXTRAS, K>();
    const size_t smem = planes_smem_bytes(S.n_planes);
    const uint64_t resident = (uint64_t)L.sm_count * pool_blocks(MB, T), need = (R.n_tuples + T - 1) / T;
    const unsigned grid = (unsigned)(need < resident ? need : resident);
    const ParkOut out1{L.park1, L.cap1, L.counts}, out2{L.park2, L.cap2, L.counts + 1}, none{nullptr, 0, nullptr};
    k_trace_pool<EXTRAS, K, MB><<<grid, T, smem + camera_smem_bytes(S.n_planes), stream>>>(
        S, B, R, xyz, L.work, L.alone ? none : out1, L.cap_first);
    if (L.alone) return;
    k_trace_resume<EXTRAS, K, MB><<<grid, T, smem, stream>>>(S, B, L.park1, L.cap1, L.counts, L.cap_second, L.work + 1,
                                                             out2, xyz);
    k_trace_resume<EXTRAS, K, MB><<<grid, T, smem, stream>>>(S, B, L.park2, L.cap2, L.counts + 1, 0xFFFFFFFFu, L.work + 2,
                                                             none, xyz);
}

}  // namespace grd
