"""Gain media: materials whose absorption or path scale is negative.  Their Stokes vectors
grow by up to e^88 a segment and leave the finite range after two, where the Mueller
products without their zero terms differ from the full ones (0 * inf is NaN, and a NaN
intensity counts as none), so such scenes run the kernels that form every term: the same
samples as with a far frosted plane, which moves any scene to those kernels, and non-finite
where the oracle's are.  Losses of the same size stay finite in either kernel."""
from __future__ import annotations

import numpy as np
import pytest

from gemray_studio_b200 import abi, scene as S, workloads as W
from helpers import oracle_trace_samples

pytestmark = pytest.mark.gpu

W_PX, H_PX, SPP = 29, 23, 24


def _scene(kind: str, frosted_far: bool = False) -> S.Scene:
    planes = np.concatenate([S.round_brilliant_57(), np.asarray([[0.6, 0.8, 0.0, -50.0]], np.float32)])
    fin = np.zeros(len(planes), np.uint32)
    fin[-1] = 1 if frosted_far else 0
    ext = None
    if kind == "table":
        mat, ext = W.birefringent_emerald_material()
        for i in range(ext.n_absorption):
            ext.alpha_o_table[i] = ext.alpha_e_table[i] = -500.0
    else:
        mat = S.builtin_material("Tourmaline")
        peak = {"bands -50": -50.0, "bands -1e4": -1e4, "path scale": 50.0, "bands 1e4": 1e4}[kind]
        for bands, n in ((mat.o_ray_bands, mat.o_ray_band_count), (mat.e_ray_bands, mat.e_ray_band_count)):
            for i in range(n):
                bands[i].peak = peak
        if kind == "path scale":
            mat.absorption_path_scale = -1.0
    return S.Scene(width=W_PX, height=H_PX, planes=planes, material=mat, cam=S.camera(0.4, 0.5, 4.0, 26.0), max_bounces=32,
                   env_mode=abi.GR_ENV_STUDIO, ext=ext, finishes=fin)


@pytest.mark.parametrize("kind", ["bands -50", "bands -1e4", "table", "path scale", "bands 1e4"])
def test_gain_media_run_the_full_sums(renderer, oracle, kind):
    n = W_PX * H_PX
    x = renderer.trace_samples(_scene(kind), 0, n, 5, SPP)
    y = renderer.trace_samples(_scene(kind, frosted_far=True), 0, n, 5, SPP)
    assert np.array_equal(np.isnan(x), np.isnan(y))
    assert np.array_equal(np.nan_to_num(x).view(np.uint32), np.nan_to_num(y).view(np.uint32))
    st, ref, _b, _t = oracle_trace_samples(oracle, _scene(kind), 0, n, 5, SPP)
    assert st == abi.GR_OK
    # as many paths may take another event than the oracle's as the parity tests allow: 1%
    assert np.mean(np.isfinite(x).all(axis=1) == np.isfinite(ref).all(axis=1)) >= 0.99
