"""The pooled transport kernels (blocks that run each bounce together, pack their live paths
and refill) and the interior plane scan, against the plain kernel and the clip in f32.

Films of the pooled and the plain kernel are bit-identical at every size where a pool can go
wrong: fewer tuples than threads, one more or one less than a block, many refills, ragged
last blocks, paths that outlive the drain's limit and are parked (depth 4096), for each block
size (clear isotropic stones 256 threads, others and the extension kernels 512).  The scan
decides most rays from approximate quotients and must still return the facet and distance of
the reference loop bit for bit: rays from inside near faces, edges and corners."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from gemray_studio_b200 import GpuFrameRenderer, abi, scene as S

pytestmark = pytest.mark.gpu


def _scene(kind: str, w: int, h: int, depth: int) -> S.Scene:
    mat = S.builtin_material({"clear": "Diamond", "general": "Tourmaline", "extras": "Tanzanite"}[kind])
    planes = S.standard_round_brilliant()
    fin = (np.abs(planes[:, 1]) < 0.05).astype(np.uint32) if kind == "extras" else None
    if kind == "extras":
        mat.scattering_sigma_s, mat.scattering_g = 0.2, 0.5
    return S.Scene(width=w, height=h, planes=planes, material=mat, cam=S.camera(0.4, 0.5, 4.0, 26.0), max_bounces=depth,
                   env_mode=abi.GR_ENV_STUDIO, finishes=fin)


@pytest.fixture(scope="module")
def pair(engine_lib):
    a, b = GpuFrameRenderer(kernel=abi.GR_KERNEL_STAGED), GpuFrameRenderer(kernel=abi.GR_KERNEL_PLAIN)
    yield a, b
    a.close()
    b.close()


SIZES = [(1, 1, 1), (255, 1, 1), (16, 16, 1), (257, 1, 1), (73, 7, 1), (16, 32, 1), (27, 19, 1), (37, 29, 13), (64, 40, 160)]


@pytest.mark.parametrize("kind", ["clear", "general", "extras"])
@pytest.mark.parametrize("size", SIZES)
def test_pool_is_the_plain_kernel(pair, kind, size):
    w, h, spp = size
    films = []
    for r in pair:
        acc = np.full((w * h, 3), 0.5, np.float32)
        r.accumulate(_scene(kind, w, h, 32), 3, spp, acc)
        films.append(acc)
    assert np.array_equal(films[0].view(np.uint32), films[1].view(np.uint32))


@pytest.mark.parametrize("kind", ["clear", "general", "extras"])
@pytest.mark.parametrize("size", [(1, 1, 3), (37, 64, 4), (37, 65, 4), (74, 65, 4), (148, 65, 4), (128, 64, 16), (128, 128, 16)])
def test_auto_small_launches_are_the_pool(pair, engine_lib, kind, size):
    """AUTO's choices below its staged size: 4, 8, 16 or 32 paths per warp (2,368 tuples a
    path), the pool alone from 2^17 (extension kernels) and 2^18 tuples (general classes)."""
    w, h, spp = size
    auto = GpuFrameRenderer()
    films = []
    for r in (auto, pair[0]):
        acc = np.full((w * h, 3), 0.25, np.float32)
        r.accumulate(_scene(kind, w, h, 24), 5, spp, acc)
        films.append(acc)
    auto.close()
    assert np.array_equal(films[0].view(np.uint32), films[1].view(np.uint32))


@pytest.mark.parametrize("kind", ["clear", "general", "extras"])
@pytest.mark.parametrize("planes", [1, 2, 511, 512])
def test_pool_with_few_and_most_planes(pair, kind, planes):
    """The camera's table: one-sided plane sets (rays that never leave), odd lists, the plane
    limit (the most shared memory), and a camera inside the stone or on one of its planes."""
    for cam in (S.camera(0.4, 0.5, 4.0, 26.0), S.camera(0.4, 0.5, 0.1, 40.0), S.camera(0.0, np.pi / 2, 1.0, 40.0)):
        films = []
        for r in pair:
            sc = _scene(kind, 24, 17, 12)
            far = np.tile(np.asarray([[0.6, 0.8, 0.0, -50.0]], np.float32), (512, 1))
            sc.planes = np.concatenate([sc.planes, far])[:planes]
            if planes < 3:
                sc.planes[0] = (0.0, 1.0, 0.0, -1.0)  # the last camera sits on this plane
            sc.cam = cam
            if sc.finishes is not None:
                sc.finishes = np.zeros(len(sc.planes), np.uint32)
            acc = np.zeros((24 * 17, 3), np.float32)
            r.accumulate(sc, 0, 9, acc)
            films.append(acc)
        assert np.array_equal(films[0].view(np.uint32), films[1].view(np.uint32))


@pytest.mark.parametrize("kind", ["clear", "general"])
def test_paths_past_the_drain_limit(pair, kind):
    """Depth 4096 in a uniform environment: the longest paths are parked and resumed."""
    films = []
    for r in pair:
        sc = _scene(kind, 48, 48, 4096)
        sc.env_mode = abi.GR_ENV_UNIFORM
        acc = np.zeros((48 * 48, 3), np.float32)
        r.accumulate(sc, 0, 64, acc)
        films.append(acc)
    assert np.array_equal(films[0].view(np.uint32), films[1].view(np.uint32))


def _clip(planes, o, d):
    """The reference clip, f32 operation for f32 operation, over all planes."""
    n, w = planes[:, :3], planes[:, 3]
    den = (d[:, 0:1] * n[:, 0] + d[:, 1:2] * n[:, 1]) + d[:, 2:3] * n[:, 2]
    side = w + ((o[:, 0:1] * n[:, 0] + o[:, 1:2] * n[:, 1]) + o[:, 2:3] * n[:, 2])
    with np.errstate(divide="ignore", invalid="ignore"):
        t = (-side / den).astype(np.float32)
    near = np.where(den < np.float32(-1e-7), t, np.float32(-1e30))
    far = np.where(den > np.float32(1e-7), t, np.float32(1e30))
    outside = ((np.abs(den) <= np.float32(1e-7)) & (side > 0)).any(axis=1)
    tn, tf, ni, fi = near.max(axis=1), far.min(axis=1), near.argmax(axis=1), far.argmin(axis=1)
    hit_n = tn > np.float32(1e-4)
    miss = outside | (tn > tf) | (~hit_n & ~(tf > np.float32(1e-4)))
    return np.where(miss, np.float32(0), np.where(hit_n, tn, tf)), np.where(miss, -1, np.where(hit_n, ni, fi))


@pytest.mark.parametrize("stone", ["srb", "rb57", "em49", "random17", "random145", "random145+512"])
def test_interior_scan_is_the_reference_clip(renderer, stone):
    rng = np.random.default_rng(11)
    if stone.startswith("random"):
        n = 17 if stone == "random17" else 145
        planes = S.random_polyhedron(rng, n_min=n, n_max=n)
        if stone.endswith("512"):  # the index's last bit: far planes up to the limit
            planes = np.concatenate([np.tile(np.asarray([[0.0, 1.0, 0.0, -40.0]], np.float32), (512 - len(planes), 1)), planes])
    else:
        planes = {"srb": S.standard_round_brilliant, "rb57": S.round_brilliant_57, "em49": S.emerald_cut_49}[stone]()
    n = 60_000
    d = rng.normal(size=(n, 3))
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
    o = np.zeros((n, 3), np.float32)
    t, f = _clip(planes, o, d)
    # origins along those rays: anywhere, close to the face, and bounced along the face toward its edges
    frac = np.concatenate([rng.uniform(0, 0.99, n // 3), 1 - 10 ** rng.uniform(-6, -1, n - n // 3)]).astype(np.float32)
    o2 = (o + (t * frac)[:, None] * d).astype(np.float32)
    along = d - (d * planes[f, :3]).sum(axis=1, keepdims=True) * planes[f, :3] * rng.uniform(0.9, 1.4, (n, 1)).astype(np.float32)
    d2 = np.where(rng.uniform(size=(n, 1)) < 0.5, along, rng.normal(size=(n, 3)))
    d2 = (d2 / np.maximum(np.linalg.norm(d2, axis=1, keepdims=True), 1e-20)).astype(np.float32)
    rays = np.concatenate([np.concatenate([o, d], 1), np.concatenate([o2, d2], 1), np.concatenate([o2 * np.float32(1.4), d2], 1)])
    rays = np.ascontiguousarray(rays, np.float32)
    ref_t, ref_f = _clip(planes, rays[:, :3], rays[:, 3:])
    got_t, got_f = np.empty(len(rays), np.float32), np.empty(len(rays), np.int32)
    p = np.ascontiguousarray(planes, np.float32)
    assert renderer.lib.gr_intersect_rays(renderer.ctx, p.ctypes.data, len(p), rays.ctypes.data_as(C.POINTER(C.c_float)),
                                          len(rays), got_t.ctypes.data_as(C.POINTER(C.c_float)),
                                          got_f.ctypes.data_as(C.POINTER(C.c_int32))) == abi.GR_OK
    assert np.array_equal(got_f, ref_f)
    assert np.array_equal(got_t.view(np.uint32), ref_t.view(np.uint32))
