"""Planes whose normals are near the largest float: a ray's denominator overflows, the
reference clip takes t = -side / inf = 0, and the ray misses.  The scans that order planes
by approximate keys have no key for an infinite quotient, so such plane sets (and rays with
such directions) take the general scan everywhere: the clip itself, the transport (events
and samples), the guide images and the metrics, each against its reference."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from gemray_studio_b200 import GpuFrameRenderer, abi, metrics as M, scene as S
from gemray_studio_b200.denoise import GuideBuffers, generate_guide_buffers
from helpers import oracle_trace_samples

pytestmark = pytest.mark.gpu

# a diagonal plane met from inside the stone, and one through the camera's axis (the camera
# at (0, 0, 5) stands 2e-6 inside of it, so the camera's keys are multiplied by 5e5)
HUGE = {"met inside": (3e38, 3e38, 0.0, -2e38), "beside the camera": (3e38, -3e38, 0.0, -2e-6)}


def _planes(kind: str) -> np.ndarray:
    return np.concatenate([S.standard_round_brilliant(), np.asarray([HUGE[kind]], np.float32)])


def _scene(kind: str, **kw) -> S.Scene:
    return S.Scene(width=40, height=30, planes=_planes(kind), material=S.builtin_material("Diamond"),
                   cam=S.camera(0.0, 0.0, 5.0, 26.0), max_bounces=12, env_mode=abi.GR_ENV_STUDIO, **kw)


def _clip(planes, o, d):
    """The reference clip of one ray, f32 operation for f32 operation."""
    f = np.float32
    near, far, ni, fi = f(-1e30), f(1e30), -1, -1
    with np.errstate(all="ignore"):
        for i, p in enumerate(planes):
            den = (p[0] * d[0] + p[1] * d[1]) + p[2] * d[2]
            side = p[3] + ((p[0] * o[0] + p[1] * o[1]) + p[2] * o[2])
            if abs(den) > f(1e-7):
                t = -side / den
                if den < 0:
                    if t > near:
                        near, ni = t, i
                elif t < far:
                    far, fi = t, i
            elif side > 0:
                return f(0), -1
    if near > far:
        return f(0), -1
    if near > f(1e-4):
        return near, ni
    return (far, fi) if far > f(1e-4) else (f(0), -1)


def test_clip(renderer):
    rng = np.random.default_rng(4)
    planes = np.concatenate([S.standard_round_brilliant(), np.asarray([HUGE["met inside"]], np.float32)])
    d = rng.normal(size=(1500, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    d[:300] = np.asarray([0.6, 0.6, 0.5]) + 0.05 * rng.normal(size=(300, 3))  # dx + dy > 1.13: the denominator overflows
    d[300:600] *= 10.0 ** rng.uniform(30, 38.4, (300, 1))  # directions near the largest float
    o = rng.uniform(-0.2, 0.2, (1500, 3))
    rays = np.ascontiguousarray(np.concatenate([o, d], 1), np.float32)
    for p in (planes, planes[:-1]):
        p = np.ascontiguousarray(p, np.float32)
        t, f = np.empty(1500, np.float32), np.empty(1500, np.int32)
        assert renderer.lib.gr_intersect_rays(renderer.ctx, p.ctypes.data, len(p), rays.ctypes.data_as(C.POINTER(C.c_float)),
                                              1500, t.ctypes.data_as(C.POINTER(C.c_float)),
                                              f.ctypes.data_as(C.POINTER(C.c_int32))) == abi.GR_OK
        ref = [_clip(p, r[:3], r[3:]) for r in rays]
        assert np.array_equal(f, np.asarray([i for _, i in ref], np.int32))
        assert np.array_equal(t.view(np.uint32), np.asarray([x for x, _ in ref], np.float32).view(np.uint32))


@pytest.mark.parametrize("frosted", [False, True])
@pytest.mark.parametrize("kind", list(HUGE))
def test_transport(engine_lib, oracle, kind, frosted):
    """The plain and the pooled kernel, with the bars of an isotropic stone."""
    sc = _scene(kind, finishes=np.eye(1, 75, 10, dtype=np.uint32)[0] if frosted else None)
    n = sc.width * sc.height
    st, ref, _b, _t = oracle_trace_samples(oracle, sc, 0, n, 0, 8)
    assert st == abi.GR_OK
    for kernel in (abi.GR_KERNEL_PLAIN, abi.GR_KERNEL_STAGED):
        r = GpuFrameRenderer(kernel=kernel)
        got = r.trace_samples(sc, 0, n, 0, 8)
        r.close()
        rel = np.abs(got - ref).max(axis=1) / np.maximum(np.abs(ref).max(axis=1), 1e-30)
        assert np.mean(rel <= 1e-5) >= 0.98 and np.mean(rel > 1e-3) <= 0.01


@pytest.mark.parametrize("kind", list(HUGE))
def test_guide_images(renderer, oracle, kind):
    sc = _scene(kind)
    n, fp = sc.width * sc.height, C.POINTER(C.c_float)
    ref = GuideBuffers(np.empty(n, np.float32), np.empty((n, 3), np.float32), np.empty(n, np.int32))
    oracle.gro_guide_buffers(C.byref(sc.c_scene()), ref.depth.ctypes.data_as(fp), ref.normal.ctypes.data_as(fp),
                             ref.facet_id.ctypes.data_as(C.POINTER(C.c_int32)))
    got = generate_guide_buffers(renderer, sc)
    assert np.array_equal(got.facet_id, ref.facet_id)
    assert got.depth.tobytes() == ref.depth.tobytes()


def test_metrics(renderer, oracle):
    planes, mat = np.ascontiguousarray(_planes("met inside")), S.builtin_material("Diamond")
    poses = np.asarray([[0.3, 0.5, 0.8, 0.9], [1.9, 0.2, 0.1, 0.7], [-2.2, 0.9, 0.4, 1.0]], np.float32)
    got = M.evaluate_poses(renderer, planes, mat, poses)
    for g, pose in zip(got, poses):
        ref = (C.c_float * 5)()
        oracle.gro_metrics(planes.ctypes.data_as(C.POINTER(abi.gr_plane)), len(planes), C.byref(mat), *map(float, pose), ref)
        ref = np.asarray(ref, np.float32)
        assert np.array_equal(g[[0, 2, 3, 4]].view(np.uint32), ref[[0, 2, 3, 4]].view(np.uint32))
        assert abs(g[1] - ref[1]) <= 1e-5 * abs(ref[1])
