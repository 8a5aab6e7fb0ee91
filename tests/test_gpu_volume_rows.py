"""Volume counts where a warp packs 16, 8, 4, 2 rows or one at a time: widths at
the edges between them, row counts that leave a warp partly empty."""

import numpy as np
import pytest

from bone_morphometry_gb300 import volume_metrics
from test_gpu_volume_counts import counts

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w", [2, 15, 16, 17, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 513])
@pytest.mark.parametrize("h,d", [(2, 2), (5, 3), (17, 9), (64, 33)])
def test_rows_per_warp(gpu_ctx, w, h, d):
    import torch

    rng = np.random.default_rng(w * h + d)
    bone = (rng.random((d, h, w)) < 0.6).astype(np.uint8) * np.uint8(255)
    roi = (rng.random((d, h, w)) < 0.9).astype(np.uint8)
    bone.flat[0] = roi.flat[0] = 1
    m = volume_metrics(torch.from_numpy(bone).cuda(), torch.from_numpy(roi).cuda(), 1.0, ctx=gpu_ctx)
    assert (m.bone_voxels, m.roi_voxels, m.boundary_bone_voxels) == counts(bone, roi)
