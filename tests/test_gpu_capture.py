"""Device memory of renders, and renders captured into a CUDA graph: AUTO's launches below its staged size allocate nothing
once the context's XYZ scratch has their size, whichever kernel they take (the plain one, or
from 2^17 / 2^18 tuples the pool alone), and a captured one stays valid after a larger staged
render has made the context grow its park buffer.  A staged launch takes park slots only
where its depth lets a path outlive the drain limit."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest
import torch

from gemray_studio_b200 import GpuFrameRenderer, abi, scene as S

pytestmark = pytest.mark.gpu


def _scene(material: str, w: int, h: int) -> S.Scene:
    sc = S.Scene(width=w, height=h, planes=S.standard_round_brilliant(), material=S.builtin_material(material),
                 cam=S.camera(0.35, 0.28, 3.0, 18.0), max_bounces=8, env_mode=abi.GR_ENV_STUDIO)
    if material == "Tanzanite":
        sc.finishes = (np.abs(sc.planes[:, 1]) < 0.05).astype(np.uint32)
    return sc


def _upload(r, sc) -> int:
    sid = C.c_uint64()
    assert r.lib.gr_scene_upload(r.ctx, C.byref(sc.c_scene()), C.byref(sid)) == abi.GR_OK
    return sid.value


@pytest.mark.parametrize("material,w,h", [("Diamond", 512, 512), ("Tourmaline", 512, 512), ("Tanzanite", 512, 256),
                                          ("Tanzanite", 64, 64)])
def test_small_launches_can_be_captured(engine_lib, material, w, h):
    n = w * h
    plain = GpuFrameRenderer(kernel=abi.GR_KERNEL_PLAIN)
    want = np.zeros((n, 3), np.float32)
    plain.accumulate(_scene(material, w, h), 4, 1, want)
    plain.close()

    r = GpuFrameRenderer()
    film = torch.zeros((n, 3), dtype=torch.float32, device="cuda")
    sid, big = _upload(r, _scene(material, w, h)), _upload(r, _scene(material, 1024, 1024))
    frame = torch.zeros((1 << 20, 3), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    assert r.lib.gr_set_kernel(r.ctx, abi.GR_KERNEL_PLAIN) == abi.GR_OK  # the XYZ scratch at its largest size here
    assert r.lib.gr_render_resident(r.ctx, big, 0, 1, frame.data_ptr(), None) == abi.GR_OK
    assert r.lib.gr_set_kernel(r.ctx, abi.GR_KERNEL_AUTO) == abi.GR_OK
    r.synchronize()
    graph, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(graph, stream=s):
        st = r.lib.gr_render_resident(r.ctx, sid, 4, 1, film.data_ptr(), C.c_void_p(s.cuda_stream))
    assert st == abi.GR_OK, r.lib.gr_last_error_string()
    for staged_before in (False, True):
        if staged_before:  # the context's first staged launch: its park buffer grows
            assert r.lib.gr_render_resident(r.ctx, big, 0, 1, frame.data_ptr(), None) == abi.GR_OK
            r.synchronize()
        film.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert np.array_equal(film.cpu().numpy().view(np.uint32), want.view(np.uint32))
    del graph
    for i in (sid, big):
        r.lib.gr_scene_release(r.ctx, i)
    r.close()


def test_a_shallow_staged_launch_takes_no_park_slots(engine_lib):
    """2^19 tuples at depth 32: the XYZ scratch (6 MiB) and counters.  A captured one stays
    valid when a deep render makes the context allocate its park buffer."""
    r = GpuFrameRenderer()
    shallow, deep = _scene("Tourmaline", 1024, 512), _scene("Tourmaline", 1024, 512)
    shallow.max_bounces, deep.max_bounces = 32, 512
    n = 1024 * 512
    a, b = _upload(r, shallow), _upload(r, deep)
    for i in (a, b):  # no schedule trials
        assert r.lib.gr_scene_set_schedule(r.ctx, i, 12, 20, 12) == abi.GR_OK
    film = torch.zeros((n, 3), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    assert r.lib.gr_render_resident(r.ctx, a, 0, 1, film.data_ptr(), None) == abi.GR_OK
    r.synchronize()
    want = film.cpu().numpy()
    assert free - torch.cuda.mem_get_info()[0] < 32 << 20
    graph, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(graph, stream=s):
        st = r.lib.gr_render_resident(r.ctx, a, 0, 1, film.data_ptr(), C.c_void_p(s.cuda_stream))
    assert st == abi.GR_OK, r.lib.gr_last_error_string()
    assert r.lib.gr_render_resident(r.ctx, b, 0, 1, film.data_ptr(), None) == abi.GR_OK
    r.synchronize()
    film.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert np.array_equal(film.cpu().numpy().view(np.uint32), want.view(np.uint32))
    del graph
    r.lib.gr_scene_release(r.ctx, a)
    r.lib.gr_scene_release(r.ctx, b)
    r.close()
