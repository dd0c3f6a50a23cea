"""The A-Trous filter's packed records against the oracle where a tap can go wrong: images one
pixel wide or high, sizes around the 32 x 8 tile, non-finite colours and depths, zero normals,
and a cosine power on each code path (64: six squarings known at compile time, other powers of
two, powf).  Tolerance: expf and powf are within 2 ULP of the oracle's glibc forms, so a tap's
weight within 8, and 25 positive weights' mean within 1e-5 relative (the bound of the filter's
other tests)."""
from __future__ import annotations

import numpy as np
import pytest

from denoise_fixtures import irregular_scene
from gemray_studio_b200.denoise import AtrousParams, GuideBuffers, denoise
from test_oracle_denoise import run as oracle_denoise

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("power", [64.0, 32.0, 1.0, 10.5])
@pytest.mark.parametrize("w,h", [(1, 70), (70, 1), (31, 7), (32, 8), (33, 9), (65, 17)])
def test_edges_and_special_values(renderer, oracle, w, h, power):
    color, depth, normal, facet = irregular_scene(w, h, 0x51ED270B + w)
    n = w * h
    color[n // 3] = (np.nan, 0.5, 0.25)
    color[n // 2] = (0.5, np.inf, 0.25)
    depth[n // 5] = np.inf
    normal[n // 7] = 0.0
    normal[n // 4] = (np.nan, 0.0, 0.0)
    normal[n // 6: n // 6 + 3] = normal[n // 6]
    p = AtrousParams(num_passes=3, normal_power=power)
    got = denoise(renderer, color, GuideBuffers(depth, normal, facet), w, h, 2, p)
    ref = oracle_denoise(oracle, color, depth, normal, facet, w, h, 2,
                         (p.num_passes, p.sigma_color, p.sigma_depth, p.normal_power, p.taper_reference_spp,
                          p.taper_identity_epsilon))
    fine = np.isfinite(ref)
    assert np.array_equal(fine, np.isfinite(got)) and np.array_equal(np.isnan(ref), np.isnan(got))
    err = np.abs(got[fine].astype(np.float64) - ref[fine]) / np.maximum(np.abs(ref[fine]), 1e-3)
    assert err.size == 0 or err.max() <= 1e-5
