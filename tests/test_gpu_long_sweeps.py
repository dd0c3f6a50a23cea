"""Metric sweeps of any length in bounded scratch: poses are traced and reduced 2,048 at a time.
A sweep's rows are those of its poses evaluated a few at a time, on either side of the
slices' edges, and the scratch stops growing at 240 MB."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from gemray_studio_b200 import GpuFrameRenderer, metrics as M, scene as S

pytestmark = pytest.mark.gpu


def _poses(n: int) -> np.ndarray:
    rng = np.random.default_rng(n)
    return rng.uniform([-3.0, 0.0, -3.0, 0.2], [3.0, 1.4, 3.0, 1.3], (n, 4)).astype(np.float32)


@pytest.mark.parametrize("n", [2047, 2048, 2049, 4097])
def test_slices_of_a_sweep(renderer, n):
    planes, mat, poses = S.round_brilliant_57(), S.builtin_material("Diamond"), _poses(n)
    whole = M.evaluate_poses(renderer, planes, mat, poses)
    parts = np.concatenate([M.evaluate_poses(renderer, planes, mat, poses[i:i + 500]) for i in range(0, n, 500)])
    assert np.array_equal(np.asarray(whole).view(np.uint32), parts.view(np.uint32))


def test_scratch_of_a_long_sweep(engine_lib):
    r = GpuFrameRenderer()
    planes, mat = S.round_brilliant_57(), S.builtin_material("Quartz")
    M.evaluate_poses(r, planes, mat, _poses(1))
    free = torch.cuda.mem_get_info()[0]
    M.evaluate_poses(r, planes, mat, _poses(5000))
    used = free - torch.cuda.mem_get_info()[0]
    r.close()
    assert used < 256 << 20
