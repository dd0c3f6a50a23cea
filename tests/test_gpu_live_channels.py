"""The default transport kernels skip the channels that chromatic termination has ended and
the colour integral of samples that add nothing; the extension kernels (frosted facets,
scattering, biaxial materials, scenes outside the finite range) take every channel every
time.  A far plane that no ray reaches, marked frosted, moves a scene to the extension
kernels without changing its paths, so both must give the same samples bit for bit: clear
and absorbing, isotropic and birefringent stones, every environment kind, black and
non-finite map texels, spans of bounce counts.  A scene outside the finite range is sent to
the extension kernels whatever its finishes."""
from __future__ import annotations

import numpy as np
import pytest

from gemray_studio_b200 import abi, scene as S, workloads as W

pytestmark = pytest.mark.gpu


def _map(texel=None) -> np.ndarray:
    m = S.gaussian_blob_latlong(64, 32, 5, seed=2)
    m[16:] = 0.0  # black below the horizon
    if texel is not None:
        m[3:9, ::5] = texel
    return m


def _scene(stone: str, material: str, env: int, depth: int, latlong=None, frosted_far=False, **kw) -> S.Scene:
    planes = {"rb57": S.round_brilliant_57, "em49": S.emerald_cut_49}[stone]()
    planes = np.concatenate([planes, np.asarray([[0.6, 0.8, 0.0, -50.0]], np.float32)])
    ext = None
    if material == "dichroic emerald":
        mat, ext = W.birefringent_emerald_material()
    elif material == "crown glass":
        mat = W.material_tables()[0][1]
    else:
        mat = S.builtin_material(material)
    fin = np.zeros(len(planes), np.uint32)
    fin[-1] = 1 if frosted_far else 0
    return S.Scene(width=29, height=23, planes=planes, material=mat, cam=S.camera(0.4, 0.5, 4.0, 26.0), max_bounces=depth,
                   env_mode=env, latlong=latlong, ext=ext, finishes=fin, **kw)


CASES = {
    "clear studio": ("rb57", "Diamond", abi.GR_ENV_STUDIO, 32, None),
    "clear map": ("rb57", "Diamond", abi.GR_ENV_LATLONG, 64, _map()),
    "clear map, infinite texels": ("rb57", "Diamond", abi.GR_ENV_LATLONG, 12, _map(np.inf)),
    "clear map, NaN texels": ("rb57", "Spinel", abi.GR_ENV_LATLONG, 12, _map(np.nan)),
    "clear uniform, one bounce": ("rb57", "Spinel", abi.GR_ENV_UNIFORM, 1, None),
    "tinted glass map": ("em49", "crown glass", abi.GR_ENV_LATLONG, 32, _map()),
    "dichroic studio": ("em49", "dichroic emerald", abi.GR_ENV_STUDIO, 64, None),
    "pleochroic uniform": ("rb57", "Tourmaline", abi.GR_ENV_UNIFORM, 4096, None),
    "uniaxial studio": ("rb57", "Zircon", abi.GR_ENV_STUDIO, 6, None),
}


@pytest.mark.parametrize("name", list(CASES))
def test_live_channels_give_the_full_sums(renderer, name):
    stone, material, env, depth, latlong = CASES[name]
    a = _scene(stone, material, env, depth, latlong)
    b = _scene(stone, material, env, depth, latlong, frosted_far=True)
    n = a.width * a.height
    x = renderer.trace_samples(a, 0, n, 5, 24)
    y = renderer.trace_samples(b, 0, n, 5, 24)
    assert np.array_equal(np.isnan(x), np.isnan(y))
    assert np.array_equal(np.nan_to_num(x).view(np.uint32), np.nan_to_num(y).view(np.uint32))
    assert np.nan_to_num(x, posinf=0.0).max() > 0.0


@pytest.mark.parametrize("index", [1.0, 1.0002, 1.005, 0.7, 9.0])
def test_indices_at_and_outside_the_range_match_the_oracle(renderer, oracle, index):
    """All but 1.005 run the extension kernels; the bars are those of an isotropic stone."""
    from helpers import oracle_trace_samples
    sc = _scene("rb57", "Diamond", abi.GR_ENV_STUDIO, 16)
    sc.material = S.custom_material(index, 0.0, 0.0)
    d = sc.material.dispersion
    d.param_a[0], d.param_a[1] = index, 0.0
    sc.material.o_ray_band_count = sc.material.e_ray_band_count = 0
    n = sc.width * sc.height
    gpu = renderer.trace_samples(sc, 0, n, 0, 8)
    st, ref, _b, _t = oracle_trace_samples(oracle, sc, 0, n, 0, 8)
    assert st == abi.GR_OK
    rel = np.abs(gpu - ref).max(axis=1) / np.maximum(np.abs(ref).max(axis=1), 1e-30)
    assert np.mean(rel <= 1e-5) >= 0.98 and np.mean(rel > 1e-3) <= 0.01
