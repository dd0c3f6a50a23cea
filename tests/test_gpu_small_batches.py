"""Batched launches of few tuples run in the plain form, one path per thread (below 2^18 tuples,
2^16 for extension scenes, where no path is deep enough to be parked).  Their films are the
plain kernel's bit for bit at the edges of a warp's lanes and of both forms, as the first call
of a context too, captured and not; and a batch of one thumbnail costs what its render does."""
from __future__ import annotations

import ctypes as C
import time

import numpy as np
import pytest
import torch

from gemray_studio_b200 import GpuFrameRenderer, abi, scene as S

pytestmark = pytest.mark.gpu

CUBE = np.asarray([[a, b, c, -0.7] for s in (1, -1) for a, b, c in ((s, 0, 0), (0, s, 0), (0, 0, s))], np.float32)


def _scene(kind: str, w: int, h: int, depth: int = 24) -> S.Scene:
    mat = {"cube": "Quartz", "clear": "Diamond", "general": "Tourmaline", "extras": "Tanzanite", "full": "Spinel"}[kind]
    sc = S.Scene(width=w, height=h, planes=CUBE if kind == "cube" else S.standard_round_brilliant(),
                 material=S.builtin_material(mat), cam=S.camera(0.35, 0.28, 5.0, 18.0), max_bounces=depth,
                 env_mode=abi.GR_ENV_STUDIO if kind != "full" else abi.GR_ENV_UNIFORM)
    if kind == "extras":
        sc.finishes = (np.abs(sc.planes[:, 1]) < 0.05).astype(np.uint32)
    if kind == "full":  # beyond the bound of the default kernels
        sc.uniform_rgb = (1e16, 1.0, 1.0)
    return sc


def _upload(r, sc) -> int:
    sid = C.c_uint64()
    assert r.lib.gr_scene_upload(r.ctx, C.byref(sc.c_scene()), C.byref(sid)) == abi.GR_OK
    return sid.value


def _batch(r, scenes, spp: int, flags: int = 0):
    films = [torch.zeros((sc.width * sc.height, 3), dtype=torch.float32, device="cuda") for sc in scenes]
    items, ids = (abi.gr_batch_item * len(scenes))(), [_upload(r, sc) for sc in scenes]
    for i, (sid, f) in enumerate(zip(ids, films)):
        items[i] = abi.gr_batch_item(sid, f.data_ptr(), 3, spp)
    torch.cuda.synchronize()
    for _ in range(2 if flags else 1):  # the second call replays the first one's graph
        for f in films:
            f.zero_()
        torch.cuda.synchronize()
        assert r.lib.gr_render_batch(r.ctx, items, len(scenes), flags, None) == abi.GR_OK, r.lib.gr_last_error_string()
        r.synchronize()
    for sid in ids:
        r.lib.gr_scene_release(r.ctx, sid)
    return [f.cpu().numpy() for f in films]


@pytest.fixture(scope="module")
def plain(engine_lib):
    r = GpuFrameRenderer(kernel=abi.GR_KERNEL_PLAIN)
    yield r
    r.close()


# (kind, sizes, spp, depth): one tuple; several segments at each count of lanes; both forms' edge
CASES = {
    "one tuple": ([("clear", 1, 1)], 1, 24),
    "four lanes, all classes": ([(k, 7 + i, 5) for i, k in enumerate(("cube", "clear", "general", "extras", "full"))], 3, 24),
    "sixteen lanes": ([("clear", 31, 37), ("clear", 29, 16)], 16, 24),
    "thirty-two lanes": ([("general", 61, 67)] * 2, 9, 24),
    "general below": ([("general", 511, 256), ("general", 511, 257)], 1, 24),
    "general at": ([("general", 512, 256)] * 2, 1, 24),
    "extras below": ([("extras", 255, 257)], 1, 24),
    "extras at": ([("extras", 256, 256)], 1, 24),
    "full": ([("full", 90, 91), ("full", 3, 2)], 5, 24),
    "deep": ([("clear", 24, 20), ("clear", 9, 9)], 8, 512),
    "no bounces": ([("general", 5, 3)], 4, 0),
}


@pytest.mark.parametrize("flags", [0, abi.GR_BATCH_GRAPH])
@pytest.mark.parametrize("name", list(CASES))
def test_films_are_the_plain_kernels(plain, name, flags):
    parts, spp, depth = CASES[name]
    scenes = [_scene(k, w, h, depth) for k, w, h in parts]
    r = GpuFrameRenderer()  # its first call
    got = _batch(r, scenes, spp, flags)
    r.close()
    for sc, film in zip(scenes, got):
        want = np.zeros((sc.width * sc.height, 3), np.float32)
        plain.accumulate(sc, 3, spp, want)
        assert np.array_equal(film.view(np.uint32), want.view(np.uint32))


def test_a_thumbnail_costs_what_its_render_does(engine_lib):
    """16 x 16 at 8 spp of a quartz cube: a batch of one 1.0 times the render, 2.2 in the pool."""
    r = GpuFrameRenderer()
    sid, film = _upload(r, _scene("cube", 16, 16)), torch.zeros((256, 3), dtype=torch.float32, device="cuda")
    items = (abi.gr_batch_item * 1)(abi.gr_batch_item(sid, film.data_ptr(), 3, 8))
    torch.cuda.synchronize()
    best = [1e9, 1e9]
    for _ in range(25):
        for k, call in enumerate((lambda: r.lib.gr_render_batch(r.ctx, items, 1, abi.GR_BATCH_GRAPH, None),
                                  lambda: r.lib.gr_render_resident(r.ctx, sid, 3, 8, film.data_ptr(), None))):
            t0 = time.perf_counter()
            assert call() == abi.GR_OK
            r.synchronize()
            best[k] = min(best[k], time.perf_counter() - t0)
    r.lib.gr_scene_release(r.ctx, sid)
    r.close()
    assert best[0] < 1.6 * best[1], best
