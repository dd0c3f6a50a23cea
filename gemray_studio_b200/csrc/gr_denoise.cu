// gr_denoise.cu -- the denoiser's guide pass and the edge-avoiding A-Trous filter.
//
// Guide pass (apps/diagram-gui/src/bridge/guide_pass.rs, generate_guide_buffers): one
// thread per pixel casts the primary ray through the pixel's corner (zero jitter) at
// the stone, through the transport kernels' plane scan, and writes (t, hit normal,
// facet index) or (1e6, 0, -1) on a miss.
//
// A-Trous (crates/gemray/src/renderer/denoise/mod.rs:154-690): 1..8 passes of a 5x5 B3
// spline kernel dilated by 2^pass, each tap gated by facet identity, a normal cosine
// power, a depth term and a colour term whose sigma tapers with the sample count; a
// pass is one thread per output pixel reading the previous pass's image (L2-resident:
// a 1080p image and its guides are ~60 MB).  Tap arithmetic follows atrous_pixel
// (:383-444) operation for operation; the depth and colour terms call CUDA's expf.
#include <cuda_runtime.h>

#include <cmath>
#include <cstring>
#include <utility>

#include "gr_ctx.h"
#include "gr_launch.cuh"

using grh::fail;

namespace grd {

// A grid of resident blocks strides over the pixels, so each block stages the planes and the
// camera's table once.
__global__ void __launch_bounds__(128) k_guide_pass(SceneConst S, const float4 *__restrict__ gplanes,
                                                    float *__restrict__ depth, float *__restrict__ normal,
                                                    int32_t *__restrict__ facet) {
    extern __shared__ float4 s_planes[];
    Planes PL = stage_plane_set(s_planes, gplanes, S.n_planes);
    PL.small = S.small_planes != 0;
    const V3 o = ld3(S.cam_o);
    stage_camera_table(PL, s_planes + planes_smem_bytes(S.n_planes) / sizeof(float4), o);
    const uint64_t n_px = (uint64_t)S.width * S.height, step = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n_px; i += step) {
        const uint32_t y = (uint32_t)(i / S.width), x = (uint32_t)(i - (uint64_t)y * S.width);
        const float aspect = S.width_f / S.height_f;
        const float u = (((float)x + 0.0f) / S.width_f - 0.5f) * 2.0f * aspect * S.fov_tan;
        const float v = (0.5f - ((float)y + 0.0f) / S.height_f) * 2.0f * S.fov_tan;
        const V3 dir = normalize(add(add(ld3(S.cam_f), mul(ld3(S.cam_r), u)), mul(ld3(S.cam_u), v)));
        float t = 0.0f;
        int idx = -1;
        float d = 1.0e6f;
        V3 n = v3(0.f, 0.f, 0.f);
        int32_t f = -1;
        int r = intersect_camera<true>(PL, dir, o, t, idx);
        if (r == SCAN_UNDECIDED) r = intersect<false>(PL, o, dir, t, idx) ? SCAN_HIT : SCAN_MISS;
        if (r == SCAN_HIT) {
            d = t;
            if (idx >= 0) {  // an empty plane set hits at t = 1e30 with the zero normal, facet 0
                const float4 p = PL.aos[idx];
                n = v3(p.x, p.y, p.z);
            }
            f = idx >= 0 ? idx : 0;
        }
        depth[i] = d;
        normal[3 * i + 0] = n.x;
        normal[3 * i + 1] = n.y;
        normal[3 * i + 2] = n.z;
        facet[i] = f;
    }
}

__device__ __forceinline__ float sanitize(float v) { return isfinite(v) ? v : 0.0f; }

// The filter's per-pixel records, so that a tap is two 16-byte loads: colour and facet id,
// unit normal and finite depth (unit_normal_or_zero, :268-276; the depth term sanitizes its
// input).  The colour is the averaged image, or the film scaled (accum * (1 / count) in
// denoise_and_tonemap_frame).  plain != NULL: the colour alone, for the identity filter.
__global__ void __launch_bounds__(256) k_denoise_prep(const float *__restrict__ normal, const float *__restrict__ depth,
                                                      const int32_t *__restrict__ facet, const float *__restrict__ film,
                                                      float4 *__restrict__ color, float4 *__restrict__ guide,
                                                      float *__restrict__ plain, float inv_count, uint32_t scale,
                                                      uint64_t n_px) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_px) return;
    V3 c = v3(film[3 * i], film[3 * i + 1], film[3 * i + 2]);
    if (scale) c = mul(c, inv_count);
    if (plain) {
        plain[3 * i + 0] = c.x;
        plain[3 * i + 1] = c.y;
        plain[3 * i + 2] = c.z;
        return;
    }
    const V3 n = v3(sanitize(normal[3 * i]), sanitize(normal[3 * i + 1]), sanitize(normal[3 * i + 2]));
    const float l = sqrtf(dot(n, n));
    const bool z = l <= 1.0e-8f;
    color[i] = make_float4(c.x, c.y, c.z, __int_as_float(facet[i]));
    guide[i] = make_float4(z ? 0.0f : n.x / l, z ? 0.0f : n.y / l, z ? 0.0f : n.z / l, sanitize(depth[i]));
}

// cos_pow (:294-311): repeated squaring for power-of-two integer exponents, else powf.
// SQ: the number of squarings where it is known at compile time (the default power 64: 6).
template <int SQ> __device__ __forceinline__ float cos_pow(float base, float power, uint32_t squarings, bool pow2) {
    if (SQ > 0) {
        float v = base;
#pragma unroll
        for (int k = 0; k < SQ; ++k) v *= v;
        return v;
    }
    if (pow2) {
        float v = base;
        for (uint32_t k = 0; k < squarings; ++k) v *= v;
        return v;
    }
    return powf(base, power);
}

struct AtrousConst {
    uint32_t w, h;
    float nisd, nits, power;
    uint32_t squarings, pow2;
};

// One pass, a thread per output pixel, 32 x 8 pixels per block (the rows of the block's taps
// overlap in L1).  Bound by issue: ~25 taps of ~60 instructions, two of them accurate expf.
// Separate 12-byte colour and normal images, depth and facet loads and 64-bit index
// arithmetic took 275 us a pass at 1920x1080, the two records per tap 163.  A tap of the
// centre's own normal (one facet of the stone) takes the centre's cosine power again.
// LAST: the output is the 12-byte image.
template <int SQ, bool LAST>
__global__ void __launch_bounds__(256) k_atrous_pass(AtrousConst A, const float4 *__restrict__ src,
                                                     const float4 *__restrict__ guide, float4 *__restrict__ dst,
                                                     float *__restrict__ out, int stride) {
    const uint32_t across = (A.w + 31u) / 32u, tile = blockIdx.x / across;
    const uint32_t x = (blockIdx.x - tile * across) * 32u + (threadIdx.x & 31u), y = tile * 8u + (threadIdx.x >> 5);
    if (x >= A.w || y >= A.h) return;
    const float B3[5] = {1.0f / 16.0f, 1.0f / 4.0f, 3.0f / 8.0f, 1.0f / 4.0f, 1.0f / 16.0f};
    const uint64_t c = (uint64_t)y * A.w + x;
    const float4 c4 = src[c], g4 = guide[c];
    const V3 scc = v3(sanitize(c4.x), sanitize(c4.y), sanitize(c4.z));
    const V3 cn = v3(g4.x, g4.y, g4.z);
    const bool cn_zero = cn.x == 0.0f && cn.y == 0.0f && cn.z == 0.0f;
    const float wn_own =
        cn_zero ? 1.0f : cos_pow<SQ>(fmaxf(clampf(dot(cn, cn), -1.0f, 1.0f), 0.0f), A.power, A.squarings, A.pow2 != 0);
    const int32_t cf = __float_as_int(c4.w);
    V3 sum = v3(0.f, 0.f, 0.f);
    float wsum = 0.0f;
#pragma unroll
    for (int ky = 0; ky < 5; ++ky) {
        const int64_t sy = (int64_t)y + (ky - 2) * stride;
        if (sy < 0 || sy >= (int64_t)A.h) continue;
        const float4 *row = src + (uint64_t)sy * A.w, *grow = guide + (uint64_t)sy * A.w;
#pragma unroll
        for (int kx = 0; kx < 5; ++kx) {
            const int64_t sx = (int64_t)x + (kx - 2) * stride;
            if (sx < 0 || sx >= (int64_t)A.w) continue;
            const float4 q4 = row[sx];
            if (__float_as_int(q4.w) != cf) continue;  // facet_weight 0: the tap is skipped
            const float4 p4 = grow[sx];
            const float kw = B3[ky] * B3[kx];
            const V3 qn = v3(p4.x, p4.y, p4.z);
            float wn = wn_own;
            if (qn.x != cn.x || qn.y != cn.y || qn.z != cn.z)
                wn = (cn_zero || (qn.x == 0.0f && qn.y == 0.0f && qn.z == 0.0f))
                         ? 1.0f
                         : cos_pow<SQ>(fmaxf(clampf(dot(cn, qn), -1.0f, 1.0f), 0.0f), A.power, A.squarings, A.pow2 != 0);
            const float wd = expf(fabsf(g4.w - p4.w) * A.nisd);
            const V3 qc = v3(q4.x, q4.y, q4.z);
            V3 sq = qc;
            if (!(fabsf(qc.x) + fabsf(qc.y) + fabsf(qc.z) < 3.0e38f))  // a component may not be finite
                sq = v3(sanitize(qc.x), sanitize(qc.y), sanitize(qc.z));
            const V3 dc = sub(scc, sq);
            const float wc = expf(dot(dc, dc) * A.nits);
            const float wgt = ((kw * wn) * wd) * wc;  // kernel_w * wf * wn * wd * wc with wf = 1
            sum = add(sum, mul(qc, wgt));
            wsum = wsum + wgt;
        }
    }
    const V3 r = wsum > 1.0e-8f ? v3(sum.x / wsum, sum.y / wsum, sum.z / wsum) : v3(c4.x, c4.y, c4.z);
    if (LAST) {
        out[3 * c + 0] = r.x;
        out[3 * c + 1] = r.y;
        out[3 * c + 2] = r.z;
    } else {
        dst[c] = make_float4(r.x, r.y, r.z, c4.w);
    }
}

}  // namespace grd

namespace {

gr_atrous_params default_params() {  // AtrousParams::default (:210-221)
    gr_atrous_params p;
    p.num_passes = 5;
    p.sigma_color = 0.35f;
    p.sigma_depth = 0.1f;
    p.normal_power = 64.0f;
    p.taper_reference_spp = 4.0f;
    p.taper_identity_epsilon = 0.02f;
    return p;
}

// The filter on device buffers; color_in is either the averaged image or (film,
// inv_count) to be scaled first.  out may alias neither input.
gr_status atrous_device(gr_ctx *ctx, const float *color_in, const float *film, float inv_count, const float *depth,
                        const float *normal, const int32_t *facet, uint32_t w, uint32_t h, uint32_t spp,
                        const gr_atrous_params *params_in, float *out, cudaStream_t s) {
    const uint64_t n_px = (uint64_t)w * h;
    if (n_px == 0) return GR_OK;
    const gr_atrous_params P = params_in ? *params_in : default_params();
    const size_t img = (size_t)n_px * 3 * sizeof(float);
    const float n0 = P.taper_reference_spp > 1.0e-8f ? P.taper_reference_spp : 1.0e-8f;
    const float taper = 1.0f / sqrtf(1.0f + (float)spp / n0);  // taper_strength (:244-250)
    const size_t records = (size_t)n_px * sizeof(float4);
    const unsigned threads = 256;
    const unsigned blocks = (unsigned)((n_px + threads - 1) / threads);
    gr_status st = ctx->dn_a.reserve(records);
    if (st == GR_OK) st = ctx->dn_b.reserve(records);
    if (st == GR_OK) st = ctx->dn_n.reserve(records);
    if (st != GR_OK) return st;
    float4 *a = (float4 *)ctx->dn_a.ptr, *b = (float4 *)ctx->dn_b.ptr, *guide = (float4 *)ctx->dn_n.ptr;
    const bool identity = taper < P.taper_identity_epsilon;  // the identity short-circuit: a plain copy
    grd::k_denoise_prep<<<blocks, threads, 0, s>>>(normal, depth, facet, film ? film : color_in, a, guide,
                                                   identity ? out : nullptr, inv_count, film ? 1u : 0u, n_px);
    GR_CUDA(cudaGetLastError());
    if (identity) return GR_OK;
    const uint32_t passes = P.num_passes < 1 ? 1 : (P.num_passes > 8 ? 8 : P.num_passes);
    const float sce = fmaxf(P.sigma_color * taper, 0.0f);
    const float sd = fmaxf(P.sigma_depth, 1.0e-8f);
    const float scs = fmaxf(sce * sce, 1.0e-8f);
    grd::AtrousConst A;
    A.w = w;
    A.h = h;
    A.nisd = -1.0f / sd;
    A.nits = -1.0f / (2.0f * scs);
    A.power = fmaxf(P.normal_power, 0.0f);
    A.pow2 = 0;
    A.squarings = 0;
    if (A.power == floorf(A.power) && A.power <= 4294967295.0f) {
        const uint32_t ip = (uint32_t)A.power;
        if (ip != 0 && (ip & (ip - 1)) == 0) {
            A.pow2 = 1;
            for (uint32_t k = ip; k > 1; k >>= 1) A.squarings++;
        }
    }
    const unsigned grid = (unsigned)(((w + 31ull) / 32u) * ((h + 7ull) / 8u));
    const bool six = A.pow2 && A.squarings == 6;
    for (uint32_t pass = 0; pass < passes; ++pass) {
        const int stride = 1 << pass;
        if (pass + 1 == passes) {
            if (six) grd::k_atrous_pass<6, true><<<grid, 256, 0, s>>>(A, a, guide, nullptr, out, stride);
            else grd::k_atrous_pass<0, true><<<grid, 256, 0, s>>>(A, a, guide, nullptr, out, stride);
        } else {
            if (six) grd::k_atrous_pass<6, false><<<grid, 256, 0, s>>>(A, a, guide, b, nullptr, stride);
            else grd::k_atrous_pass<0, false><<<grid, 256, 0, s>>>(A, a, guide, b, nullptr, stride);
            std::swap(a, b);
        }
        GR_CUDA(cudaGetLastError());
    }
    return GR_OK;
}

// The guide pass reads only the scene's camera, frame size and planes.  Runs on the
// context stream (its plane buffer is the context's); the caller holds ctx->mu.
gr_status guide_device(gr_ctx *ctx, const gr_scene *sc, float *depth, float *normal, int32_t *facet) {
    if (sc->n_planes > GR_MAX_PLANES) return fail(GR_EINVAL, "n_planes %u exceeds %u", sc->n_planes, GR_MAX_PLANES);
    if (sc->n_planes && !sc->planes) return fail(GR_EINVAL, "planes is NULL");
    const uint64_t n_px = (uint64_t)sc->width * sc->height;
    if (n_px == 0) return GR_OK;
    SceneConst S;
    std::memset(&S, 0, sizeof(S));
    for (int i = 0; i < 3; ++i) {
        S.cam_o[i] = sc->camera.origin[i];
        S.cam_f[i] = sc->camera.forward[i];
        S.cam_r[i] = sc->camera.right[i];
        S.cam_u[i] = sc->camera.up[i];
    }
    S.fov_tan = sc->camera.fov_tan;
    S.width = sc->width;
    S.height = sc->height;
    S.width_f = (float)sc->width;
    S.height_f = (float)sc->height;
    S.n_planes = sc->n_planes;
    S.small_planes = grh::planes_small(sc->planes, sc->n_planes);
    gr_status st = ctx->dn_planes.reserve((size_t)(sc->n_planes ? sc->n_planes : 1) * sizeof(float4));
    if (st != GR_OK) return st;
    if (sc->n_planes)
        GR_CUDA(cudaMemcpyAsync(ctx->dn_planes.ptr, sc->planes, sc->n_planes * sizeof(gr_plane), cudaMemcpyHostToDevice,
                                ctx->stream));
    const unsigned threads = 128;
    const uint64_t resident = (uint64_t)(ctx->sm_count > 0 ? ctx->sm_count : 1) * 12u, need = (n_px + threads - 1) / threads;
    grd::k_guide_pass<<<(unsigned)(need < resident ? need : resident), threads,
                        grd::planes_smem_bytes(S.n_planes) + grd::camera_smem_bytes(S.n_planes), ctx->stream>>>(
        S, (const float4 *)ctx->dn_planes.ptr, depth, normal, facet);
    GR_CUDA(cudaGetLastError());
    // the host planes are copied from pageable memory: wait before the caller may free them
    GR_CUDA(cudaStreamSynchronize(ctx->stream));
    return GR_OK;
}

// Device-pointer entry points run on the context stream (their scratch is the
// context's) ordered after the caller's stream, and the caller's stream after them.
gr_status join_in(gr_ctx *ctx, cudaStream_t user) {
    if (!user || user == ctx->stream) return GR_OK;
    if (!ctx->dn_ev) GR_CUDA(cudaEventCreateWithFlags(&ctx->dn_ev, cudaEventDisableTiming));
    GR_CUDA(cudaEventRecord(ctx->dn_ev, user));
    GR_CUDA(cudaStreamWaitEvent(ctx->stream, ctx->dn_ev, 0));
    return GR_OK;
}
gr_status join_out(gr_ctx *ctx, cudaStream_t user) {
    if (!user || user == ctx->stream) return GR_OK;
    GR_CUDA(cudaEventRecord(ctx->dn_ev, ctx->stream));
    GR_CUDA(cudaStreamWaitEvent(user, ctx->dn_ev, 0));
    return GR_OK;
}

}  // namespace

extern "C" {

gr_status gr_guide_buffers(gr_ctx *ctx, const gr_scene *sc, float *depth, float *normal, int32_t *facet_id) {
    if (!ctx || !sc) return fail(GR_EINVAL, "ctx or scene is NULL");
    const uint64_t n_px = (uint64_t)sc->width * sc->height;
    if (n_px == 0) return GR_OK;
    if (!depth || !normal || !facet_id) return fail(GR_EINVAL, "output buffer is NULL");
    std::lock_guard<std::mutex> lk(ctx->mu);
    GR_CUDA(cudaSetDevice(ctx->device));
    gr_status st = ctx->dn_g.reserve((size_t)n_px * 5 * sizeof(float));
    if (st != GR_OK) return st;
    float *dd = (float *)ctx->dn_g.ptr, *dn = dd + n_px;
    int32_t *df = (int32_t *)(dn + 3 * n_px);
    st = guide_device(ctx, sc, dd, dn, df);
    if (st != GR_OK) return st;
    GR_CUDA(cudaMemcpyAsync(depth, dd, n_px * sizeof(float), cudaMemcpyDeviceToHost, ctx->stream));
    GR_CUDA(cudaMemcpyAsync(normal, dn, n_px * 3 * sizeof(float), cudaMemcpyDeviceToHost, ctx->stream));
    GR_CUDA(cudaMemcpyAsync(facet_id, df, n_px * sizeof(int32_t), cudaMemcpyDeviceToHost, ctx->stream));
    GR_CUDA(cudaStreamSynchronize(ctx->stream));
    return GR_OK;
}

gr_status gr_guide_buffers_device(gr_ctx *ctx, const gr_scene *sc, float *depth, float *normal, int32_t *facet_id,
                                  void *stream) {
    if (!ctx || !sc) return fail(GR_EINVAL, "ctx or scene is NULL");
    if ((uint64_t)sc->width * sc->height == 0) return GR_OK;
    if (!depth || !normal || !facet_id) return fail(GR_EINVAL, "output buffer is NULL");
    std::lock_guard<std::mutex> lk(ctx->mu);
    GR_CUDA(cudaSetDevice(ctx->device));
    gr_status st = join_in(ctx, (cudaStream_t)stream);
    if (st == GR_OK) st = guide_device(ctx, sc, depth, normal, facet_id);
    if (st == GR_OK) st = join_out(ctx, (cudaStream_t)stream);
    return st;
}

gr_status gr_atrous_denoise(gr_ctx *ctx, const float *color, const float *depth, const float *normal,
                            const int32_t *facet_id, uint32_t width, uint32_t height, uint32_t spp,
                            const gr_atrous_params *params, float *out) {
    if (!ctx) return fail(GR_EINVAL, "ctx is NULL");
    const uint64_t n_px = (uint64_t)width * height;
    if (n_px == 0) return GR_OK;
    if (!color || !depth || !normal || !facet_id || !out) return fail(GR_EINVAL, "buffer is NULL");
    std::lock_guard<std::mutex> lk(ctx->mu);
    GR_CUDA(cudaSetDevice(ctx->device));
    const size_t img = (size_t)n_px * 3 * sizeof(float);
    gr_status st = ctx->dn_in.reserve(2 * img + (size_t)n_px * (sizeof(float) + sizeof(int32_t)) + img);
    if (st != GR_OK) return st;
    float *dc = (float *)ctx->dn_in.ptr, *dn = dc + 3 * n_px, *dd = dn + 3 * n_px;
    int32_t *df = (int32_t *)(dd + n_px);
    float *dout = (float *)(df + n_px);
    cudaStream_t s = ctx->stream;
    GR_CUDA(cudaMemcpyAsync(dc, color, img, cudaMemcpyHostToDevice, s));
    GR_CUDA(cudaMemcpyAsync(dn, normal, img, cudaMemcpyHostToDevice, s));
    GR_CUDA(cudaMemcpyAsync(dd, depth, n_px * sizeof(float), cudaMemcpyHostToDevice, s));
    GR_CUDA(cudaMemcpyAsync(df, facet_id, n_px * sizeof(int32_t), cudaMemcpyHostToDevice, s));
    st = atrous_device(ctx, dc, nullptr, 1.0f, dd, dn, df, width, height, spp, params, dout, s);
    if (st != GR_OK) return st;
    GR_CUDA(cudaMemcpyAsync(out, dout, img, cudaMemcpyDeviceToHost, s));
    GR_CUDA(cudaStreamSynchronize(s));
    return GR_OK;
}

gr_status gr_atrous_denoise_device(gr_ctx *ctx, const float *color, const float *depth, const float *normal,
                                   const int32_t *facet_id, uint32_t width, uint32_t height, uint32_t spp,
                                   const gr_atrous_params *params, float *out, void *stream) {
    if (!ctx) return fail(GR_EINVAL, "ctx is NULL");
    if ((uint64_t)width * height == 0) return GR_OK;
    if (!color || !depth || !normal || !facet_id || !out) return fail(GR_EINVAL, "buffer is NULL");
    if (out == color) return fail(GR_EINVAL, "out must not alias color");
    std::lock_guard<std::mutex> lk(ctx->mu);
    GR_CUDA(cudaSetDevice(ctx->device));
    gr_status st = join_in(ctx, (cudaStream_t)stream);
    if (st == GR_OK)
        st = atrous_device(ctx, color, nullptr, 1.0f, depth, normal, facet_id, width, height, spp, params, out,
                           ctx->stream);
    if (st == GR_OK) st = join_out(ctx, (cudaStream_t)stream);
    return st;
}

gr_status gr_denoise_tonemap_device(gr_ctx *ctx, const float *film, uint32_t sample_count, const float *depth,
                                    const float *normal, const int32_t *facet_id, uint32_t width, uint32_t height,
                                    const gr_atrous_params *params, void *rgba, void *stream) {
    if (!ctx) return fail(GR_EINVAL, "ctx is NULL");
    const uint64_t n_px = (uint64_t)width * height;
    if (n_px == 0) return GR_OK;
    if (!film || !depth || !normal || !facet_id || !rgba) return fail(GR_EINVAL, "buffer is NULL");
    if (n_px > 0xFFFFFFFFull) return fail(GR_EINVAL, "frame too large");
    std::lock_guard<std::mutex> lk(ctx->mu);
    GR_CUDA(cudaSetDevice(ctx->device));
    cudaStream_t s = ctx->stream;
    gr_status st = ctx->dn_out.reserve((size_t)n_px * 3 * sizeof(float));
    if (st == GR_OK) st = join_in(ctx, (cudaStream_t)stream);
    if (st != GR_OK) return st;
    const float inv = 1.0f / (float)sample_count;  // denoise.rs: 1.0 / current_sample_count as f32
    st = atrous_device(ctx, nullptr, film, inv, depth, normal, facet_id, width, height, sample_count, params,
                       (float *)ctx->dn_out.ptr, s);
    if (st == GR_OK) st = grh::tonemap_device((const float *)ctx->dn_out.ptr, 1.0f, (uint32_t)n_px, rgba, s);
    if (st == GR_OK) st = join_out(ctx, (cudaStream_t)stream);
    return st;
}

}  // extern "C"
