"""Stokes films of few tuples: launches below 2^18 tuples (2^16 for extension scenes) run the
plain kernel, larger ones the pool.  Both give the same films bit for bit, whichever sizes a
frame is cut into, and the XYZ film is gr_accumulate's; a small film does not wait for the
pool's large blocks."""
from __future__ import annotations

import ctypes as C
import time

import numpy as np
import pytest

from gemray_studio_b200 import GpuFrameRenderer, abi, scene as S

pytestmark = pytest.mark.gpu

_fp = C.POINTER(C.c_float)
CUBE = np.asarray([[a, b, c, -0.7] for s in (1, -1) for a, b, c in ((s, 0, 0), (0, s, 0), (0, 0, s))], np.float32)


def _scene(material: str, w: int, h: int) -> S.Scene:
    cube = material == "Quartz"
    sc = S.Scene(width=w, height=h, planes=CUBE if cube else S.standard_round_brilliant(),
                 material=S.builtin_material(material), cam=S.camera(0.35, 0.28, 5.0, 18.0), max_bounces=16,
                 env_mode=abi.GR_ENV_STUDIO)
    if material == "Tanzanite":
        sc.finishes = (np.abs(sc.planes[:, 1]) < 0.05).astype(np.uint32)
    return sc


def _films(r, sc, spp: int):
    n = sc.width * sc.height
    x, s = np.zeros((n, 3), np.float32), np.zeros((n, 4), np.float32)
    assert r.lib.gr_accumulate_stokes(r.ctx, C.byref(sc.c_scene()), 5, spp, x.ctypes.data_as(_fp),
                                      s.ctypes.data_as(_fp)) == abi.GR_OK
    return x, s


# one tuple; the lanes of a warp (4, 16, 32 tuples); one tuple below, at and past each limit
@pytest.mark.parametrize("material,w,h,spp", [("Quartz", 1, 1, 1), ("Diamond", 7, 5, 3), ("Diamond", 41, 29, 8), ("Tourmaline", 53, 59, 7),
                                              ("Tourmaline", 487, 538, 1), ("Tourmaline", 512, 512, 1), ("Tourmaline", 149, 353, 5),
                                              ("Tanzanite", 255, 257, 1), ("Tanzanite", 256, 256, 1), ("Tanzanite", 64, 331, 4)])
def test_plain_and_pooled_films_agree(renderer, material, w, h, spp):
    sc = _scene(material, w, h)
    x, s = _films(renderer, sc, spp)
    acc = np.zeros_like(x)
    renderer.accumulate(sc, 5, spp, acc)
    assert np.array_equal(x.view(np.uint32), acc.view(np.uint32))
    assert s.max() > 0.0
    small = GpuFrameRenderer(chunk_budget_bytes=28 * 30000)  # launches of at most 30,000 tuples: plain
    x2, s2 = _films(small, sc, spp)
    small.close()
    assert np.array_equal(x.view(np.uint32), x2.view(np.uint32)) and np.array_equal(s.view(np.uint32), s2.view(np.uint32))


def test_small_films_cost_what_small_renders_do(renderer):
    """2,048 tuples of a quartz cube: 1.12 times gr_accumulate on B200, 1.78 in the pool."""
    sc, best = _scene("Quartz", 16, 16), [1e9, 1e9]
    acc = np.zeros((256, 3), np.float32)
    for _ in range(20):
        for k, call in enumerate((lambda: _films(renderer, sc, 8), lambda: renderer.accumulate(sc, 5, 8, acc))):
            t0 = time.perf_counter()
            call()
            best[k] = min(best[k], time.perf_counter() - t0)
    assert best[0] < 1.45 * best[1], best
