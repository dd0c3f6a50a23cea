// gr_stage.cuh -- the pooled transport scheme shared by the single-scene kernels
// (gr_transport.cuh), the batched ones (gr_batch.cuh) and the Stokes film.
#pragma once

#include "gr_launch.cuh"

namespace grd {

// Pooled kernels.  A block holds T paths, one per thread, and runs each bounce together:
// scan, facet, reflections, refractions, with a barrier between them.  When half of its
// paths have ended, the live ones are packed into the low threads (records swapped through
// shared memory), the high threads -- now whole warps -- write their finished samples and
// start the launch's next ones, so a block stays full until the supply runs out.  Then it
// drains.  Paths that outlive the drain's bounce limit (DRAIN_CAPS times the schedule's cap:
// deep scenes only) are parked for the next stage, which runs the same pool over the parked
// records, packed densely.
//
// Why: a bounce is ~2,500 instructions of mostly straight code (the kernels are 60 to 110
// KB), and warps that run it each at their own place starve on instruction fetch -- on the
// dichroic emerald 18.6 of 34 cycles per issued instruction, issue slots 49% busy.  With
// barriers the block's warps fetch the same lines at the same time: 0.6 cycles, 72% busy.
// And a warp whose lanes end at different bounces idles: packing and refilling costs ~150
// instructions a swap and keeps three lanes of four on a live path.
// Measured (1080p brilliant, 1024^2 emerald at 32 spp, 317x211 tourmaline at 37, frosted
// tanzanite at 24; ms): one path per thread in 128-thread blocks, parked past caps 50.0 /
// 69.3 / 3.54 / 13.7; barriers 46.0 / 45.6 / 3.07 / 8.3; packing as well 44.0 / 44.7 / 3.2 /
// 8.1; refilling as well 43.0 / 43.8 / 2.68 / 7.4; with the paths ending at the facet they
// leave through (step_leave) 36.9 / 38.5 / 2.37 / 6.5.
// T: 512 threads align four warps of each scheduler; the clear isotropic kernels fetch less
// and wait more, so theirs are 256 (brilliant at 64 spp 71.7 against 73.2 ms, 256^2 at 64 spp
// 4.14 against 4.48).  1,024 lost on both (52.5 / 52.8 against 47.8 / 50.1 before refilling).
// Every path runs the same functions in the same order as in the plain kernel, so every
// sample is bit-identical; only its thread changes.
template <bool EXTRAS, int K> __host__ __device__ constexpr int pool_threads() {
    return (!EXTRAS && (K & K_ISO) && (K & K_CLEAR)) ? 256 : 512;
}
// Resident blocks per SM of T threads for a target given in 128-thread blocks.
__host__ __device__ constexpr int pool_blocks(int mb, int T) { return mb * 128 / T > 0 ? mb * 128 / T : 1; }

// The bounce caps of the stages where no schedule is chosen yet.
#ifndef GR_STAGE_CAP
#define GR_STAGE_CAP 12
#endif
#ifndef GR_STAGE_CAP2
#define GR_STAGE_CAP2 20
#endif

// Where a draining pool parks the paths past its cap (cap 0: nowhere, they run to their end).
struct ParkOut {
    Path *park;
    uint32_t cap;
    unsigned int *count;
};

// A draining block keeps its paths to DRAIN_CAPS times the stage's cap.  Parking them at the
// cap itself cost 0.4-0.5 ms a launch (tourmaline 2.70 against 2.39 ms, 256^2 brilliant 4.64
// against 4.21): the next stage begins its serial chain of bounces only when this one has
// ended, and the SM's other blocks hide a thin block's latency meanwhile.
constexpr uint32_t DRAIN_CAPS = 8;
// The float4 rows of a path record that the kernels of a class use.
template <bool EXTRAS, int K> __host__ __device__ constexpr uint32_t record_rows() {
    return ((!EXTRAS && (K & K_ISO) && (K & K_CLEAR)) ? PATH_CLEAR_BYTES : sizeof(Path)) / sizeof(float4);
}
template <uint32_t ROWS> __device__ __forceinline__ void copy_record(Path &dst, const Path &src) {
    float4 *d = reinterpret_cast<float4 *>(&dst);
    const float4 *s = reinterpret_cast<const float4 *>(&src);
#pragma unroll 4
    for (uint32_t r = 0; r < ROWS; ++r) d[r] = s[r];
}

// Supplies of a pool: claim(n) hands the block the next n items, [base, base + n), of which
// those below `end` exist.  PoolQueue: one counter for all blocks of the launch (64 bits:
// every block claims once past the end).  PoolRange: the block's own range.
struct PoolQueue {
    unsigned long long *next;
    uint64_t end;
    __device__ __forceinline__ void claim(uint64_t &base, uint32_t n) {
        if (threadIdx.x == 0) base = atomicAdd(next, (unsigned long long)n);
    }
};
struct PoolRange {
    uint64_t next, end;
    __device__ __forceinline__ void claim(uint64_t &base, uint32_t n) {
        if (threadIdx.x == 0) base = next;
        next += n;
    }
};

// Packs the block's n_live live paths (`go`) into threads [0, n_live): each live record past
// there swaps places with a record that has ended below it, row by row through shared memory
// (at most T / 2 pairs, so at least two rows a pass).  Called by the whole block.
template <int T, uint32_t ROWS> __device__ __forceinline__ void pack_block(Path &P, bool go, uint32_t n_live) {
    __shared__ uint32_t s_mask[T / 32];
    __shared__ float4 s_rows[2 * T];
    const uint32_t tid = threadIdx.x, w = tid >> 5;
    const uint32_t m = __ballot_sync(0xffffffffu, go);
    if ((tid & 31u) == 0) s_mask[w] = m;
    __syncthreads();
    // live paths below this thread, and below thread n_live
    uint32_t before = 0, kept = 0;
    const uint32_t wl = n_live >> 5;
#pragma unroll
    for (uint32_t i = 0; i < T / 32; ++i) {
        const uint32_t v = s_mask[i], c = __popc(v);
        if (i < w) before += c;
        if (i < wl) kept += c;
        else if (i == wl) kept += __popc(v & ((1u << (n_live & 31u)) - 1u));
    }
    before += __popc(m & ((1u << (tid & 31u)) - 1u));
    const uint32_t moves = n_live - kept;  // block-uniform
    const bool mover = go && tid >= n_live, hole = !go && tid < n_live;
    const uint32_t put = mover ? before - kept : moves + (tid - before);
    const uint32_t get = mover ? put + moves : put - moves;
    const uint32_t chunk = moves ? min(ROWS, 2u * T / (2u * moves)) : ROWS;
    float4 *row = reinterpret_cast<float4 *>(&P);
    for (uint32_t r0 = 0; r0 < ROWS && moves; r0 += chunk) {
        const uint32_t r1 = min(r0 + chunk, ROWS);
        if (mover || hole)
            for (uint32_t r = r0; r < r1; ++r) s_rows[(r - r0) * 2u * moves + put] = row[r];
        __syncthreads();
        if (mover || hole)
            for (uint32_t r = r0; r < r1; ++r) row[r] = s_rows[(r - r0) * 2u * moves + get];
        __syncthreads();
    }
}

// Runs a block's pool: `start(P, i)` begins item i of the supply in a thread's record,
// `store(P)` writes a finished path's sample.  Once the supply has run out, paths that have
// made DRAIN_CAPS * `cap` bounces are parked in `out` while it has slots.  CAM: the planes
// carry the camera's table.  Called by the whole block of T threads; every barrier is reached
// by all of them.
// Packing without a refill (the drain) waits until a quarter of the warps would be freed: a
// swap costs about a tenth of a bounce.  Refilling at three quarters instead of half a block
// measured 43.3 against 40.5 ms on the brilliant and 48.6 against 43.8 on the emerald: more
// swaps, and finishes and starts in smaller groups.
template <int T, bool EXTRAS, int K, bool CAM, class Supply, class Start, class Store>
__device__ __forceinline__ void run_pool(Path &P, const SceneConst &S, const SceneBuffers &B, const Planes &PL,
                                         Supply supply, uint32_t cap, const ParkOut &out, Start start, Store store) {
    __shared__ uint64_t s_base;
    constexpr uint32_t ROWS = record_rows<EXTRAS, K>();
    NoCounters nc;
    bool more = true;        // items may remain (block-uniform)
    uint32_t extent = T;     // live paths are in threads below (block-uniform)
    set_state_bits(P, F_NONE);
    for (;;) {
        bool go = (state_bits(P) & F_ALIVE) != 0;
        if (!more && out.cap) {
            const bool want = go && p_bounce(P) / DRAIN_CAPS >= cap;
            const uint32_t mask = __ballot_sync(0xffffffffu, want);
            if (mask) {  // warp-uniform
                const uint32_t lane = threadIdx.x & 31u, leader = __ffs((int)mask) - 1;
                uint32_t slot = 0;
                if (lane == leader) {
                    // A full buffer is not asked again: such paths come here at every bounce, and
                    // the 32-bit count has to stay below the slots plus the resident threads.
                    slot = *(volatile unsigned int *)out.count;
                    if (slot < out.cap) slot = atomicAdd(out.count, (unsigned)__popc(mask));
                }
                slot = __shfl_sync(0xffffffffu, slot, leader) + __popc(mask & ((1u << lane) - 1u));
                if (want && slot < out.cap) {  // a full buffer: the path runs on here
                    copy_record<ROWS>(out.park[slot], P);
                    set_state_bits(P, F_NONE);
                    go = false;
                }
            }
        }
        const uint32_t n_live = (uint32_t)__syncthreads_count(go);
        if (more && 2u * n_live <= (uint32_t)T) {
            const uint32_t n = T - n_live;
            supply.claim(s_base, n);
            if (n_live) pack_block<T, ROWS>(P, go, n_live);
            __syncthreads();
            const uint64_t base = s_base;
            if (threadIdx.x >= n_live) {
                if (!(state_bits(P) & F_NONE)) store(P);
                const uint64_t i = base + (threadIdx.x - n_live);
                if (i < supply.end) start(P, i);
                else set_state_bits(P, F_NONE);
            }
            more = base + n < supply.end;
            go = (state_bits(P) & F_ALIVE) != 0;
        } else if (n_live == 0) {
            break;
        } else if (!more && 4u * ((n_live + 31u) & ~31u) <= 3u * extent) {
            pack_block<T, ROWS>(P, go, n_live);
            extent = (n_live + 31u) & ~31u;
            go = threadIdx.x < n_live;
        }
        Event E;
        uint32_t ev = EV_DONE;
        float t_hit = 0.0f;
        int fidx = 0;
        const bool hit = go && step_scan<NoCounters, false, CAM>(P, PL, t_hit, fidx, nc);
        __syncthreads();
        if (hit) ev = step_facet<1, NoCounters, false, EXTRAS, K>(P, S, B, PL, t_hit, fidx, E, nc);
        __syncthreads();
        if (ev == EV_REFLECT) step_reflect<1, NoCounters, EXTRAS, K>(P, S, E, nc);
        __syncthreads();
        if (ev == EV_REFRACT) step_refract<1, NoCounters, EXTRAS, K>(P, S, E, nc);
        if (hit) step_leave(P, PL, fidx);
    }
    if (!(state_bits(P) & F_NONE)) store(P);
}

}  // namespace grd
