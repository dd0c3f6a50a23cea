// gr_metrics.cu -- brilliance / fire / scintillation / windowing / extinction out,
// = evaluate_gem_optical_metrics (crates/gemray/src/color/metrics.rs:1082-1237) for
// a batch of poses (tilt sweeps, metrics.rs:1262-1289, are batches of poses).
//
// k_metric_traces: one thread per (pose, trace, cell of the unit disc); traces 0..14 are the
//   five aperture rays of classify_aperture_sample (metrics.rs:568-676), each at the d, F
//   and C lines, traces 15..19 the d line at the five yaw offsets of cell_temporal_variance
//   (metrics.rs:349-380).  Bound by latency (a chain of up to eleven plane scans on a chip
//   that 16 poses fill to a third), so the three lines of a ray run side by side although
//   F and C only count where d returns, cells outside the disc get no thread, and the scan
//   is the transport's branch-free one.
// k_metric_reduce: one block per pose classifies the samples in parallel and then forms each
//   of the reference's f32 sums in its order (cells ix-major, then aperture order) in one
//   thread, the sums side by side in separate warps, so counts are exact and sums are formed
//   in the same sequence.
// 16 poses of the 73-plane brilliant: one thread per (pose, cell, ray) with the three lines in
// turn 746 us and one thread per pose reducing 464 us, 1.22 ms a call; now 0.19 ms a call.
// Camera bases, the studio rig and the d/F/C indices are host-computed per pose with
// the reference's f32 libm arithmetic.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "gemray_cuda.h"
#include "gr_host.h"
#include "gr_launch.cuh"

namespace grd {

constexpr int MGRID = 18;
constexpr int MAPS = 5;                    // aperture rays; as many yaw offsets
constexpr int MTRACES = 3 * MAPS + MAPS;   // per cell
constexpr int MCELLS_MAX = MGRID * MGRID;

struct PoseConst {
    float fwd[3], right[3], up[3];         // camera_view_basis(cam_yaw, cam_pitch)
    float tf[5][3], tr[5][3], tu[5][3];    // bases at the five temporal yaw offsets
    float key[3], fill[3], sin_lp;         // StudioRig::new(light_yaw, light_pitch)
    float nd, nf, nc;                      // indices at 589.3 / 486.1 / 656.3 nm
};

// One trace's end: fate 0 entry blocked, 1 leaked, 2 exited upward, 3 absorbed, 4 no hit, 5
// exited upward and visible (d-line traces).
struct __align__(16) MetricTrace {
    uint32_t fate;
    int32_t facet;
    uint32_t bounces;
    float transmittance, exit_cos, dx, dy, dz;
};

// metrics.rs:118-131
__device__ __forceinline__ float m_fresnel_t(float n1, float n2, float ci, float ct) {
    float ds = fmaf(n2, ct, n1 * ci), dp = fmaf(n2, ci, n1 * ct);
    if (fabsf(ds) < 1e-6f || fabsf(dp) < 1e-6f) return 0.0f;
    float a = fmaf(n2, -ct, n1 * ci) / ds, b = fmaf(n2, -ci, n1 * ct) / dp;
    return clampf(1.0f - midpoint(a * a, b * b), 0.0f, 1.0f);
}

struct MExit {
    V3 dir;
    float transmittance, exit_cos;
    int facet;
    uint32_t bounces;
};

// metrics.rs:138-227 (fates: 0 blocked, 1 leaked, 2 exited upward, 3 absorbed)
__device__ int m_trace_wavelength(V3 entry, V3 in_dir, V3 n_entry, float cos_i, const Planes &PL, float index,
                                  MExit &ex) {
    float sin2_t = (1.0f / (index * index)) * fmaf(cos_i, -cos_i, 1.0f);
    if (sin2_t > 1.0f) return 0;
    float cos_t = sqrtf(1.0f - sin2_t);
    V3 dir = normalize(add(smul(1.0f / index, in_dir), smul(fmaf(1.0f / index, cos_i, -cos_t), n_entry)));
    V3 hp = add(entry, mul(dir, 1e-4f));
    float sin_crit = 1.0f / index;
    float entry_t = m_fresnel_t(1.0f, index, cos_i, cos_t);
    bool leaked = false, up = false;
    for (uint32_t bounce = 0; bounce < 10; ++bounce) {
        float t = 0.0f;
        int idx = 0;
        if (!intersect_from(PL, true, hp, dir, t, idx)) break;
        V3 np = add(hp, smul(t, dir));
        V3 n_out = plane_normal(PL.aos, idx);
        float ct = clampf(dot(dir, n_out), 0.0f, 1.0f);
        float st = sqrtf(fmaxf(fmaf(ct, -ct, 1.0f), 0.0f));
        if (st < sin_crit) {
            float s2o = (index * index) * fmaf(ct, -ct, 1.0f);
            if (s2o <= 1.0f) {
                float co = sqrtf(1.0f - s2o);
                V3 od = normalize(add(smul(index, dir), smul(fmaf(index, -ct, co), n_out)));
                if (n_out.y < -0.05f) {
                    leaked = true;
                } else if (od.y > 0.05f) {
                    up = true;
                    ex.dir = od;
                    ex.transmittance = m_fresnel_t(index, 1.0f, ct, co);
                    ex.exit_cos = co;
                    ex.facet = idx < 0 ? 0 : idx;
                    ex.bounces = bounce;
                }
                break;
            }
        }
        dir = normalize(sub(dir, smul(2.0f * ct, n_out)));
        hp = add(np, mul(dir, 1e-4f));
    }
    if (leaked) return 1;
    if (up) {
        ex.transmittance = entry_t * ex.transmittance;
        return 2;
    }
    return 3;
}

// metrics.rs:229-252
__device__ __forceinline__ bool m_visible(V3 d, V3 fwd, const PoseConst &P) {
    bool head = dot(neg(d), fwd) > 0.96f;
    float kd = fmaxf(dot(d, ld3(P.key)), 0.0f), fd = fmaxf(dot(d, ld3(P.fill)), 0.0f);
    bool ring = fabsf(fmaf(P.sin_lp, -0.8f, d.y)) < 0.35f;
    bool lit = (kd > 0.70f) || (fd > 0.75f) || (ring && d.y > 0.2f);
    return !head && lit;
}

__host__ __device__ __forceinline__ bool cell_uv(int ix, int iz, float &u, float &v) {
    u = fmaf(((float)ix + 0.5f) / (float)MGRID, 2.0f, -1.0f);
    v = fmaf(((float)iz + 0.5f) / (float)MGRID, 2.0f, -1.0f);
    return !(fmaf(v, v, u * u) > 0.70f);
}

// cells: the disc's cells (ix * MGRID + iz) in the reference's order.
__global__ void __launch_bounds__(128) k_metric_traces(const PoseConst *__restrict__ poses, uint32_t n_poses,
                                                       const uint16_t *__restrict__ cells, uint32_t n_cells,
                                                       const float4 *__restrict__ gplanes, uint32_t n_planes,
                                                       uint32_t small, MetricTrace *__restrict__ out) {
    extern __shared__ float4 s_planes[];
    Planes PL = stage_plane_set(s_planes, gplanes, n_planes);
    PL.small = small != 0;
    const uint64_t gid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (gid >= (uint64_t)n_poses * MTRACES * n_cells) return;
    const uint32_t ray = (uint32_t)(gid / n_cells), cell = cells[gid - (uint64_t)ray * n_cells];
    const uint32_t pose = ray / MTRACES, trace = ray - pose * MTRACES;
    const PoseConst &P = poses[pose];
    float u, v;
    cell_uv((int)(cell / MGRID), (int)(cell % MGRID), u, v);
    const bool aperture = trace < 3 * MAPS;
    const uint32_t line = aperture ? trace % 3u : 0u, k = aperture ? trace / 3u : trace - 3u * MAPS;
    V3 ro, rd, fwd;
    if (aperture) {
        // classify_aperture_sample (metrics.rs:568-676)
        const float ap[MAPS][2] = {{0.f, 0.f}, {0.08f, 0.f}, {-0.08f, 0.f}, {0.f, 0.08f}, {0.f, -0.08f}};
        fwd = ld3(P.fwd);
        const V3 right = ld3(P.right), upv = ld3(P.up);
        rd = normalize(add(add(fwd, smul(ap[k][0], right)), smul(ap[k][1], upv)));
        ro = add(add(mul(neg(fwd), 2.5f), smul(u * 0.95f, right)), smul(v * 0.95f, upv));
    } else {
        // cell_returned_at_yaw_offset (metrics.rs:295-330)
        fwd = rd = ld3(P.tf[k]);
        ro = add(add(mul(neg(fwd), 2.5f), smul(u * 0.95f, ld3(P.tr[k]))), smul(v * 0.95f, ld3(P.tu[k])));
    }
    MetricTrace r{4u, 0, 0u, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    float t = 0.0f;
    int idx = 0;
    if (intersect<false>(PL, ro, rd, t, idx)) {
        const V3 hp = add(ro, smul(t, rd));
        const V3 nrm = plane_normal(PL.aos, idx);
        const float ci = clampf(dot(neg(rd), nrm), 0.0f, 1.0f);
        MExit e;
        r.fate = (uint32_t)m_trace_wavelength(hp, rd, nrm, ci, PL, line == 0 ? P.nd : (line == 1 ? P.nf : P.nc), e);
        if (r.fate == 2u) {
            r.facet = e.facet;
            r.bounces = e.bounces;
            r.transmittance = e.transmittance;
            r.exit_cos = e.exit_cos;
            r.dx = e.dir.x;
            r.dy = e.dir.y;
            r.dz = e.dir.z;
            if (line == 0 && m_visible(e.dir, fwd, P)) r.fate = 5u;
        }
    }
    out[gid] = r;
}

// Sample classes: 0 no hit, 1 entry blocked, 2 windowed, 3 extinct, 4 returned.
constexpr int MREDUCE_THREADS = 256;
__global__ void __launch_bounds__(MREDUCE_THREADS) k_metric_reduce(const MetricTrace *__restrict__ in, uint32_t n_cells,
                                                                   gr_metrics_out *__restrict__ out, uint32_t use_fp64) {
    __shared__ uint8_t s_cls[MCELLS_MAX * MAPS], s_fire[MCELLS_MAX * MAPS];
    __shared__ float s_angle[MCELLS_MAX * MAPS], s_weight[MCELLS_MAX * MAPS];
    __shared__ float s_frac[MCELLS_MAX], s_tv[MCELLS_MAX];
    __shared__ uint32_t s_count[5];  // samples per class, cells with a hit in [0]
    __shared__ float s_sum[4];       // fire, cell fraction, its square, temporal variance
    const MetricTrace *p = in + (size_t)blockIdx.x * MTRACES * n_cells;
    const uint32_t tid = threadIdx.x;
    if (tid < 5) s_count[tid] = 0;
    __syncthreads();
    for (uint32_t i = tid; i < n_cells * MAPS; i += MREDUCE_THREADS) {
        const uint32_t a = i / n_cells, c = i - a * n_cells, at = c * MAPS + a;  // aperture order within a cell
        const MetricTrace d = p[(3 * a) * n_cells + c];
        uint32_t cls = d.fate == 4u ? 0u : (d.fate == 0u ? 1u : (d.fate == 1u ? 2u : (d.fate == 5u ? 4u : 3u)));
        uint8_t fire = 0;
        if (cls == 4u) {
            const MetricTrace f = p[(3 * a + 1) * n_cells + c], g = p[(3 * a + 2) * n_cells + c];
            if (f.fate == 2u && g.fate == 2u && f.facet == g.facet && f.bounces == g.bounces) {
                const float cs = clampf(dot(v3(f.dx, f.dy, f.dz), v3(g.dx, g.dy, g.dz)), -1.0f, 1.0f);
                s_angle[at] = m_acos(cs) * 57.2957795130823208767981548141051703f;
                s_weight[at] = (d.transmittance * f.transmittance * g.transmittance) *
                               (fmaxf(f.exit_cos, 0.0f) * fmaxf(g.exit_cos, 0.0f));
                fire = 1;
            }
        }
        s_cls[at] = (uint8_t)cls;
        s_fire[at] = fire;
        if (cls) atomicAdd(&s_count[cls], 1u);
    }
    __syncthreads();
    for (uint32_t c = tid; c < n_cells; c += MREDUCE_THREADS) {
        uint32_t total = 0, ret = 0, tr = 0;
        for (int a = 0; a < MAPS; ++a) {
            total += s_cls[c * MAPS + a] != 0;
            ret += s_cls[c * MAPS + a] == 4;
            tr += p[(3 * MAPS + a) * n_cells + c].fate == 5u;
        }
        s_frac[c] = total ? (float)ret / (float)total : -1.0f;  // -1: no ray of the cell hit
        const float tp = (float)tr / 5.0f;
        s_tv[c] = fmaf(tp, -tp, tp);
        if (total) atomicAdd(&s_count[0], 1u);
    }
    __syncthreads();
    // The reference's accumulation order (metrics.rs:1127-1236), one sum per warp.
    if (tid == 0) {
        float fire = 0.f;
        double fire_d = 0.0;
        for (uint32_t i = 0; i < n_cells * MAPS; ++i) {
            if (!s_fire[i]) continue;
            fire = fmaf(s_angle[i], s_weight[i], fire);
            if (use_fp64) fire_d = fma((double)s_angle[i], (double)s_weight[i], fire_d);
        }
        s_sum[0] = use_fp64 ? (float)fire_d : fire;
    } else if (tid == 32) {
        float sum = 0.f;
        double sum_d = 0.0;
        for (uint32_t c = 0; c < n_cells; ++c) {
            const float f = s_frac[c];
            if (f < 0.0f) continue;
            sum += f;
            if (use_fp64) sum_d += (double)f;
        }
        s_sum[1] = use_fp64 ? (float)sum_d : sum;
    } else if (tid == 64) {
        float sq = 0.f;
        double sq_d = 0.0;
        for (uint32_t c = 0; c < n_cells; ++c) {
            const float f = s_frac[c];
            if (f < 0.0f) continue;
            sq = fmaf(f, f, sq);
            if (use_fp64) sq_d = fma((double)f, (double)f, sq_d);
        }
        s_sum[2] = use_fp64 ? (float)sq_d : sq;
    } else if (tid == 96) {
        float tv = 0.f;
        double tv_d = 0.0;
        for (uint32_t c = 0; c < n_cells; ++c) {
            if (s_frac[c] < 0.0f) continue;
            tv += s_tv[c];
            if (use_fp64) tv_d += (double)s_tv[c];
        }
        s_sum[3] = use_fp64 ? (float)tv_d : tv;
    }
    __syncthreads();
    if (tid != 0) return;
    const uint32_t windowed = s_count[2], extinct = s_count[3], returned = s_count[4], cell_count = s_count[0];
    const uint32_t total = s_count[1] + windowed + extinct + returned;
    const float cf_sum = s_sum[1], cf_sq = s_sum[2], tv_sum = s_sum[3];
    const float nt = (float)(total > 1 ? total : 1);
    gr_metrics_out o;
    o.windowing_pct = clampf((float)windowed / nt * 100.0f, 0.0f, 100.0f);
    o.extinction_pct = clampf((float)extinct / nt * 100.0f, 0.0f, 100.0f);
    o.brilliance_pct = clampf((float)returned / nt * 100.0f, 0.0f, 100.0f);
    o.fire_index = fmaxf(s_sum[0] / nt * 275.0f, 0.1f);
    float spatial = 0.0f;
    if (cell_count > 0) {
        float mean = cf_sum / (float)cell_count;
        if (mean > 1e-4f) {
            float var = fmaxf(fmaf(mean, -mean, cf_sq / (float)cell_count), 0.0f);
            float cv = sqrtf(var) / mean;
            spatial = clampf(cv / (1.0f + cv) * 100.0f, 0.0f, 100.0f);
        }
    }
    float temporal = cell_count > 0 ? clampf((tv_sum / (float)cell_count) / 0.24f * 100.0f, 0.0f, 100.0f) : 0.0f;
    o.scintillation_pct = clampf(fmaf(0.4f, temporal, 0.6f * spatial), 0.0f, 100.0f);
    out[blockIdx.x] = o;
}

}  // namespace grd

namespace {

struct H3 {
    float x, y, z;
};
inline float hdot(H3 a, H3 b) { return (a.x * b.x + a.y * b.y) + a.z * b.z; }
inline H3 hnorm(H3 a) {
    float r = 1.0f / sqrtf(hdot(a, a));
    return H3{a.x * r, a.y * r, a.z * r};
}
inline H3 hcross(H3 a, H3 b) { return H3{a.y * b.z - b.y * a.z, a.z * b.x - b.z * a.x, a.x * b.y - b.x * a.y}; }

// metrics.rs:16-30
void camera_view_basis(float yaw, float pitch, float f[3], float r[3], float u[3]) {
    float cp = cosf(pitch), sp = sinf(pitch), cy = cosf(yaw), sy = sinf(yaw);
    H3 fw = hnorm(H3{-cp * sy, -sp, -cp * cy});
    H3 wu = fabsf(cp) < 1e-4f ? H3{0.f, 0.f, -1.f} : H3{0.f, 1.f, 0.f};
    H3 rt = hnorm(hcross(fw, wu));
    H3 up = hnorm(hcross(rt, fw));
    f[0] = fw.x; f[1] = fw.y; f[2] = fw.z;
    r[0] = rt.x; r[1] = rt.y; r[2] = rt.z;
    u[0] = up.x; u[1] = up.y; u[2] = up.z;
}

float host_dispersion(const gr_dispersion &d, float lambda_nm) {  // optics/dispersion.rs:12-37
    float lum = lambda_nm * 1e-3f, l2 = lum * lum;
    if (d.model_type == GR_DISP_SELLMEIER1) return sqrtf(fmaxf(1.0f + (d.param_a[0] * l2) / (l2 - d.param_b[0]), 1.0f));
    if (d.model_type == GR_DISP_SELLMEIER3) {
        float n2 = 1.0f;
        n2 = n2 + (d.param_a[0] * l2) / (l2 - d.param_b[0]);
        n2 = n2 + (d.param_a[1] * l2) / (l2 - d.param_b[1]);
        n2 = n2 + (d.param_a[2] * l2) / (l2 - d.param_b[2]);
        return sqrtf(fmaxf(n2, 1.0f));
    }
    float l4 = l2 * l2;
    return d.param_a[0] + (d.param_a[1] / l2) + (d.param_a[2] / l4);
}

}  // namespace

namespace grh {
void studio_rig(float yaw, float pitch, float key[3], float fill[3], float ring[16][3]);

namespace {
// The disc's cells (ix * MGRID + iz) in the reference's order; returns their number.
uint32_t disc_cells(uint16_t cells[grd::MCELLS_MAX]) {
    uint32_t n = 0;
    for (int ix = 0; ix < grd::MGRID; ++ix)
        for (int iz = 0; iz < grd::MGRID; ++iz) {
            float u, v;
            if (grd::cell_uv(ix, iz, u, v)) cells[n++] = (uint16_t)(ix * grd::MGRID + iz);
        }
    return n;
}
// Poses traced and reduced at a time, so that a sweep of any length needs no more scratch than
// these: a trace is 32 bytes, a pose 115 KB of them.  The traces' tail and the reduction between
// two slices cost 67 us, and 2,048 poses take 5.4 ms: slices of 256 made 4,096 poses 11.8 ms
// instead of 10.8.
constexpr uint32_t kMetricPoses = 2048;
// The inputs (poses, cell list, planes) first, in one upload; then a slice's traces and the
// results.
struct MetricsLayout {
    uint16_t cells[grd::MCELLS_MAX];
    uint32_t n_cells;
    size_t cell_off, plane_off, in_bytes, trace_bytes, out_bytes;
    size_t total() const { return in_bytes + trace_bytes + out_bytes; }
};
size_t up256(size_t v) { return (v + 255) & ~(size_t)255; }
MetricsLayout metrics_layout(uint32_t n_planes, uint32_t n_poses) {
    MetricsLayout L;
    L.n_cells = disc_cells(L.cells);
    L.cell_off = up256((size_t)n_poses * sizeof(grd::PoseConst));
    L.plane_off = L.cell_off + up256(sizeof(L.cells));
    L.in_bytes = L.plane_off + up256((size_t)(n_planes ? n_planes : 1) * sizeof(float4));
    L.trace_bytes = up256((size_t)std::min(n_poses, kMetricPoses) * grd::MTRACES * L.n_cells * sizeof(grd::MetricTrace));
    L.out_bytes = (size_t)n_poses * sizeof(gr_metrics_out);
    return L;
}
}  // namespace

size_t metrics_scratch_bytes(uint32_t n_planes, uint32_t n_poses) { return metrics_layout(n_planes, n_poses).total(); }

gr_status metrics_device(const gr_plane *planes, uint32_t n_planes, const gr_material *m, const gr_pose *poses,
                         uint32_t n_poses, gr_metrics_out *out, uint32_t flags, cudaStream_t stream, DeviceBuffer &scratch) {
    const MetricsLayout L = metrics_layout(n_planes, n_poses);
    gr_status st = scratch.reserve(L.total());
    if (st != GR_OK) return st;
    std::vector<char> staged(L.in_bytes);
    grd::PoseConst *pc = (grd::PoseConst *)staged.data();
    std::memcpy(staged.data() + L.cell_off, L.cells, sizeof(L.cells));
    if (n_planes) std::memcpy(staged.data() + L.plane_off, planes, n_planes * sizeof(gr_plane));
    const float nd = fmaxf(host_dispersion(m->dispersion, 589.3f), 1.1f);
    const float nf = fmaxf(host_dispersion(m->dispersion, 486.1f), 1.001f);
    const float nc = fmaxf(host_dispersion(m->dispersion, 656.3f), 1.001f);
    const float yaw_off[5] = {-3.0f, -1.5f, 0.0f, 1.5f, 3.0f};
    const float deg2rad = 3.14159265358979323846f / 180.0f;
    for (uint32_t i = 0; i < n_poses; ++i) {
        grd::PoseConst &P = pc[i];
        camera_view_basis(poses[i].cam_yaw, poses[i].cam_pitch, P.fwd, P.right, P.up);
        for (int k = 0; k < 5; ++k)
            camera_view_basis(poses[i].cam_yaw + yaw_off[k] * deg2rad, poses[i].cam_pitch, P.tf[k], P.tr[k], P.tu[k]);
        float ring[16][3];
        studio_rig(poses[i].light_yaw, poses[i].light_pitch, P.key, P.fill, ring);
        P.sin_lp = sinf(poses[i].light_pitch);
        P.nd = nd;
        P.nf = nf;
        P.nc = nc;
    }
    char *base = (char *)scratch.ptr;
    grd::MetricTrace *d_traces = (grd::MetricTrace *)(base + L.in_bytes);
    gr_metrics_out *d_out = (gr_metrics_out *)(base + L.in_bytes + L.trace_bytes);
    if (cudaMemcpyAsync(base, staged.data(), L.in_bytes, cudaMemcpyHostToDevice, stream) != cudaSuccess) return GR_ECUDA;
    const unsigned T = 128;
    const uint32_t small = planes_small(planes, n_planes);
    for (uint32_t first = 0; first < n_poses; first += kMetricPoses) {
        const uint32_t n = std::min(n_poses - first, kMetricPoses), threads = n * grd::MTRACES * L.n_cells;
        grd::k_metric_traces<<<(threads + T - 1) / T, T, grd::planes_smem_bytes(n_planes), stream>>>(
            (const grd::PoseConst *)base + first, n, (const uint16_t *)(base + L.cell_off), L.n_cells,
            (const float4 *)(base + L.plane_off), n_planes, small, d_traces);
        grd::k_metric_reduce<<<n, grd::MREDUCE_THREADS, 0, stream>>>(d_traces, L.n_cells, d_out + first,
                                                                     (flags & GR_METRICS_FP64_SUMS) ? 1u : 0u);
    }
    if (cudaGetLastError() != cudaSuccess) return GR_ECUDA;
    if (cudaMemcpyAsync(out, d_out, L.out_bytes, cudaMemcpyDeviceToHost, stream) != cudaSuccess) return GR_ECUDA;
    if (cudaStreamSynchronize(stream) != cudaSuccess) return GR_ECUDA;
    return GR_OK;
}
}  // namespace grh
