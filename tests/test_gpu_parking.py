"""Parked paths: a brilliant of index 7.5 at depth 1024, a fifth of whose paths outlive the
first stage's drain limit (8 x 12 bounces) and more than a tenth the second's (8 x 20), so both
stages park and resume, and more paths than a batched segment's region holds (1/16 of its
tuples).  Films are the plain kernel's bit for bit, for each block size and record (clear,
general and the extension kernels' full records), and a region that is full is not asked for
more slots: the count passes them by the asks in flight alone, at most one per thread."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest
import torch

from gemray_studio_b200 import GpuFrameRenderer, abi, scene as S

pytestmark = pytest.mark.gpu

KINDS = ["clear", "general", "extras"]
W_PX, H_PX, SPP = 40, 32, 64
TUPLES = W_PX * H_PX * SPP


def _scene(kind: str) -> S.Scene:
    sc = S.Scene(width=W_PX, height=H_PX, planes=S.standard_round_brilliant(), material=S.custom_material(7.5, 0.0, 0.0),
                 cam=S.camera(0.35, 0.28, 3.0, 18.0), max_bounces=1024, env_mode=abi.GR_ENV_UNIFORM)
    m = sc.material
    if kind != "clear":  # a trace of absorption
        m.o_ray_band_count = m.e_ray_band_count = 1
        for b in (m.o_ray_bands[0], m.e_ray_bands[0]):
            b.center_nm, b.width_nm, b.peak = 500.0, 40.0, 1e-6
    if kind == "extras":
        sc.finishes = (np.abs(sc.planes[:, 1]) < 0.05).astype(np.uint32)
    return sc


@pytest.fixture(scope="module")
def plain_films(engine_lib):
    r = GpuFrameRenderer(kernel=abi.GR_KERNEL_PLAIN)
    films = {}
    for kind in KINDS:
        films[kind] = np.zeros((W_PX * H_PX, 3), np.float32)
        r.accumulate(_scene(kind), 0, SPP, films[kind])
    r.close()
    return films


def _parked(r, n_batch: int):
    one, many = (C.c_uint32 * 2)(), (C.c_uint32 * max(1, n_batch))()
    assert r.lib.gr_parked_counts(r.ctx, one, many, n_batch) == abi.GR_OK
    return list(one), list(many)[:n_batch]


@pytest.mark.parametrize("kind", KINDS)
def test_parked_paths_end_as_the_plain_kernels(plain_films, kind):
    r = GpuFrameRenderer(kernel=abi.GR_KERNEL_STAGED)
    acc = np.zeros((W_PX * H_PX, 3), np.float32)
    r.accumulate(_scene(kind), 0, SPP, acc)
    (first, second), _ = _parked(r, 0)
    r.close()
    assert np.array_equal(acc.view(np.uint32), plain_films[kind].view(np.uint32))
    assert TUPLES // 8 < first <= 2 * TUPLES and TUPLES // 32 < second <= 2 * TUPLES


@pytest.mark.parametrize("kinds", [["clear"], ["general"], ["extras"], ["general", "general"], KINDS])
def test_full_batch_regions(plain_films, kinds):
    r = GpuFrameRenderer()
    ids, films = [], [torch.zeros((W_PX * H_PX, 3), dtype=torch.float32, device="cuda") for _ in kinds]
    items = (abi.gr_batch_item * len(kinds))()
    for i, kind in enumerate(kinds):
        sid = C.c_uint64()
        assert r.lib.gr_scene_upload(r.ctx, C.byref(_scene(kind).c_scene()), C.byref(sid)) == abi.GR_OK
        ids.append(sid.value)
        items[i] = abi.gr_batch_item(sid.value, films[i].data_ptr(), 0, SPP)
    torch.cuda.synchronize()
    assert r.lib.gr_render_batch(r.ctx, items, len(kinds), 0, None) == abi.GR_OK
    _, counts = _parked(r, len(kinds) if len(set(kinds)) == 1 else 1)  # classes are launched one after another
    for f, kind in zip(films, kinds):
        assert np.array_equal(f.cpu().numpy().view(np.uint32), plain_films[kind].view(np.uint32))
    for c in counts:
        assert TUPLES // 16 + 32 <= c <= TUPLES // 16 + 32 + TUPLES  # full: the last ask may fit exactly
    for i in ids:
        r.lib.gr_scene_release(r.ctx, i)
    r.close()
