// gr_launch.cuh -- launch-shape helpers shared by the transport kernels: the tuple
// numbering of a launch, shared-memory staging of the facet planes and the ordered
// per-pixel film fold.
//
// Work unit: a tuple t in [0, n_pixels * spp) of one launch maps to
//   pixel = first_pixel + t / spp, absolute sample = sample_offset + t % spp,
// the reference kernel's `idx = pixel * spp + s` numbering
// (renderer/shaders/spectral_transport.wgsl:672-691), and its XYZ lands in
// xyz[3 * t .. 3 * t + 3), whatever the order in which a launch takes its tuples (pooled
// launches take a pixel's samples in HeroOrder from 64 on).  The fold then sums each pixel's spp samples in sample
// order and adds the sum once to the film -- the reference's per-pixel
// `sum += sample; accum[p] += sum` (renderer/gpu/frame.rs:799-814).
#pragma once

#include "gr_trace.cuh"

namespace grd {

constexpr int TRACE_THREADS = 128;

struct LaunchRange {
    uint32_t first_pixel;
    uint32_t n_pixels;
    uint32_t sample_offset;
    uint32_t spp;
    uint64_t n_tuples;  // n_pixels * spp
};

// Both shared-memory layouts of the paired scan (planes_smem_bytes(n) bytes at sp).
__device__ __forceinline__ Planes stage_plane_set(float4 *sp, const float4 *__restrict__ gp, uint32_t n) {
    float4 *pairs = sp + n;
    const uint32_t np = (n + 1u) >> 1;
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) sp[i] = gp[i];
    for (uint32_t j = threadIdx.x; j < np; j += blockDim.x) {
        const float4 a = gp[2 * j];
        const float4 b = 2 * j + 1 < n ? gp[2 * j + 1] : make_float4(0.0f, 0.0f, 0.0f, -1.0f);
        pairs[2 * j] = make_float4(a.x, b.x, a.y, b.y);
        pairs[2 * j + 1] = make_float4(a.z, b.z, a.w, b.w);
    }
    __syncthreads();
    return Planes{sp, pairs, n};
}
// The planes of a scene: the extension kernels and those of class K_FULL take scenes of any
// planes, the others small planes.
template <bool X, int K = K_ANY>
__device__ __forceinline__ Planes stage_scene_planes(float4 *sp, const SceneConst &S, const SceneBuffers &B) {
    Planes PL = stage_plane_set(sp, B.planes, S.n_planes);
    if (X || (K & K_FULL)) PL.small = S.small_planes != 0;
    PL.cam_inside = S.cam_inside != 0;
    return PL;
}

// The camera's table of the staged planes (intersect_camera) at ct, camera_smem_bytes(n):
// built by the first warp, one plane per lane; the whole block calls.
__device__ __forceinline__ void stage_camera_table(Planes &PL, float4 *ct, V3 o) {
    if (threadIdx.x < 32u) {
        const uint32_t lane = threadIdx.x;
        auto side_of = [&](uint32_t i) {
            const float4 p = PL.aos[i];
            return p.w + ((p.x * o.x + p.y * o.y) + p.z * o.z);
        };
        uint32_t n1 = 0, bad = PL.small ? 0u : 1u;
        float min1 = 3.0e38f, min2 = 3.0e38f;
        for (uint32_t b = 0; b < PL.n; b += 32u) {
            const bool on = b + lane < PL.n;
            const float s = on ? side_of(b + lane) : -1.0f;
            bad |= __ballot_sync(0xffffffffu, on && !(fabsf(s) >= 1e-6f && fabsf(s) < 1e15f));
            n1 += __popc(__ballot_sync(0xffffffffu, on && s > 0.0f));
            if (on && s > 0.0f) min1 = fminf(min1, s);
            else if (on) min2 = fminf(min2, -s);
        }
        for (int k = 16; k; k >>= 1) {
            min1 = fminf(min1, __shfl_xor_sync(0xffffffffu, min1, k));
            min2 = fminf(min2, __shfl_xor_sync(0xffffffffu, min2, k));
        }
        const uint32_t n2 = PL.n - n1, p1 = (n1 + 1u) / 2u, p2 = p1 + (n2 + 1u) / 2u;
        if (lane == 0)
            ct[0] = make_float4(__uint_as_float(bad ? 0u : p1), __uint_as_float(p2), 1.001e-7f / min1, 1.001e-7f / min2);
        float *f = reinterpret_cast<float *>(ct + 1);
        auto put = [&](uint32_t pair, uint32_t half, float4 p, float rs, float bias, uint32_t i) {
            float *e = f + 12u * pair + half;
            e[0] = p.x;
            e[2] = p.y;
            e[4] = p.z;
            e[6] = rs;
            e[8] = bias;
            e[10] = __uint_as_float(i);
        };
        uint32_t c1 = 0;
        for (uint32_t b = 0; b < PL.n && !bad; b += 32u) {
            const uint32_t i = b + lane;
            const bool on = i < PL.n;
            const float s = on ? side_of(i) : -1.0f;
            const uint32_t m = __ballot_sync(0xffffffffu, on && s > 0.0f), below = (1u << lane) - 1u;
            const uint32_t r1 = c1 + __popc(m & below), r2 = i - r1;
            if (on && s > 0.0f) put(r1 / 2u, r1 & 1u, PL.aos[i], -1.0f / s, 0.0f, i);
            else if (on) put(p1 + r2 / 2u, r2 & 1u, PL.aos[i], -1.0f / s, 0.0f, i);
            c1 += __popc(m);
        }
        const float4 none = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (lane == 0 && !bad && (n1 & 1u)) put(p1 - 1u, 1u, none, 0.0f, 3.0e38f, 0u);
        if (lane == 0 && !bad && (n2 & 1u)) put(p2 - 1u, 1u, none, 0.0f, -3.0e38f, 0u);
    }
    PL.cam = ct;
    __syncthreads();
}

__device__ __forceinline__ void tuple_coords(const LaunchRange &R, uint64_t t, uint32_t &pixel, uint32_t &sample) {
    uint32_t local_pixel = (uint32_t)(t / R.spp);
    uint32_t s = (uint32_t)(t - (uint64_t)local_pixel * R.spp);
    pixel = R.first_pixel + local_pixel;
    sample = R.sample_offset + s;  // u32 wrapping add, as the reference's wrapping_add
}


// A finished path's sample into its tuple's place.
__device__ __forceinline__ void store_sample(float *__restrict__ xyz, const Path &P, V3 c) {
    const uint64_t t = p_tuple(P);
    xyz[3 * t + 0] = c.x;
    xyz[3 * t + 1] = c.y;
    xyz[3 * t + 2] = c.z;
}

// The order in which a pooled launch takes a pixel's samples: by hero wavelength, whose
// leading base-5 digits are the low digits of the sample index (sampling.rs:170-181), in 25
// classes of 16 nm.  Chromatic termination leaves neighbouring heroes the same number of live
// channels, and a warp runs its channel loops as often as its richest path: 288.8 -> 275.1 ms
// on the 1080p brilliant at 256 spp, 144.6 -> 140.7 at 128, 4.23 -> 4.16 at 256^2 and 64 spp,
// 36.9 -> 37.0 at 32 spp, so from 64 samples on; 64 batched stones of 32 to 512 spp 27.5 ->
// 26.7.  Grouping the classes over several pixels lost more than it gained (38.9 ms at 32 spp).
constexpr uint32_t HERO_CLASSES = 25, HERO_MIN_SPP = 64;
struct HeroOrder {
    uint32_t first[HERO_CLASSES + 1];  // samples of one pixel before class k
    uint32_t residue[HERO_CLASSES];    // class k: samples residue, residue + 25, ...
};
// Filled by the block, for a launch of at least HERO_MIN_SPP samples.
__device__ __forceinline__ void hero_order(HeroOrder &H, const LaunchRange &R) {
    if (threadIdx.x == 0) {
        const uint32_t off = R.sample_offset % HERO_CLASSES;
        uint32_t at = 0;
        for (uint32_t k = 0; k < HERO_CLASSES; ++k) {
            const uint32_t r = (k / 5u + 5u * (k % 5u) + HERO_CLASSES - off) % HERO_CLASSES;  // digits reversed
            H.first[k] = at;
            H.residue[k] = r;
            at += (R.spp - r - 1u) / HERO_CLASSES + 1u;
        }
        H.first[HERO_CLASSES] = at;
    }
    __syncthreads();
}
// The launch's i-th path in that order: its pixel and sample within the launch's ranges.  A
// permutation of each pixel's samples, whatever the offset (which may wrap).
__device__ __forceinline__ void hero_coords(const LaunchRange &R, const HeroOrder &H, uint64_t i, uint32_t &px, uint32_t &s) {
    px = (uint32_t)(i / R.spp);
    s = (uint32_t)(i - (uint64_t)px * R.spp);
    if (R.spp < HERO_MIN_SPP) return;
    uint32_t k = 0;  // the last class that begins at or before s
#pragma unroll
    for (uint32_t step = 16; step; step >>= 1)
        if (k + step < HERO_CLASSES && H.first[k + step] <= s) k += step;
    s = H.residue[k] + HERO_CLASSES * (s - H.first[k]);
}

// One warp folds pixel `px` (local to its xyz block) into film pixel `film_pixel`.
// Add mode (cont == 0): the samples are summed in order from zero and the sum is
// added to the film once -- the reference's per-call semantics.  Continue mode
// (cont != 0): the sum starts from the film's current value (and, with Kahan, from
// the compensation kept in comp) and is written back, so successive slices of one
// sample range on a zero film form exactly one sequential sum, whatever the slicing.
__device__ __forceinline__ void fold_pixel(const float *__restrict__ xyz, uint64_t px, uint32_t spp, uint32_t film_pixel,
                                           float *__restrict__ film, uint32_t kahan, uint32_t cont = 0,
                                           float *__restrict__ comp = nullptr) {
    const uint32_t lane = threadIdx.x & 31u;
    const float *src = xyz + (size_t)px * spp * 3;
    const size_t p = (size_t)film_pixel * 3;
    float sx = 0.0f, sy = 0.0f, sz = 0.0f;
    float cx = 0.0f, cy = 0.0f, cz = 0.0f;
    if (cont) {
        sx = film[p + 0];
        sy = film[p + 1];
        sz = film[p + 2];
        if (kahan) {
            cx = comp[p + 0];
            cy = comp[p + 1];
            cz = comp[p + 2];
        }
    }
    for (uint32_t s0 = 0; s0 < spp; s0 += 32) {
        uint32_t s = s0 + lane;
        float x = 0.f, y = 0.f, z = 0.f;
        if (s < spp) {
            x = src[3 * s + 0];
            y = src[3 * s + 1];
            z = src[3 * s + 2];
        }
        uint32_t cnt = spp - s0 < 32u ? spp - s0 : 32u;
        for (uint32_t j = 0; j < cnt; ++j) {
            float vx = __shfl_sync(0xffffffffu, x, j);
            float vy = __shfl_sync(0xffffffffu, y, j);
            float vz = __shfl_sync(0xffffffffu, z, j);
            if (kahan) {
                float yx = vx - cx, tx = sx + yx; cx = (tx - sx) - yx; sx = tx;
                float yy = vy - cy, ty = sy + yy; cy = (ty - sy) - yy; sy = ty;
                float yz = vz - cz, tz = sz + yz; cz = (tz - sz) - yz; sz = tz;
            } else {
                sx = sx + vx;
                sy = sy + vy;
                sz = sz + vz;
            }
        }
    }
    if (lane == 0) {
        if (cont) {
            film[p + 0] = sx;
            film[p + 1] = sy;
            film[p + 2] = sz;
            if (kahan) {
                comp[p + 0] = cx;
                comp[p + 1] = cy;
                comp[p + 2] = cz;
            }
        } else {
            film[p + 0] = film[p + 0] + sx;
            film[p + 1] = film[p + 1] + sy;
            film[p + 2] = film[p + 2] + sz;
        }
    }
}

}  // namespace grd
