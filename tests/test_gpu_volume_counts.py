"""Volume counts at ragged sizes and alignments (whole numbers: compared for equality)."""

import numpy as np
import pytest

from bone_morphometry_gb300 import volume_metrics

pytestmark = pytest.mark.gpu


def counts(bone, roi):
    b, r = (bone != 0) & (roi != 0), roi != 0
    p = np.pad(r, 1)
    inner = p[:-2, 1:-1, 1:-1] & p[2:, 1:-1, 1:-1] & p[1:-1, :-2, 1:-1] & p[1:-1, 2:, 1:-1] & p[1:-1, 1:-1, :-2] & \
        p[1:-1, 1:-1, 2:]
    return int(b.sum()), int(r.sum()), int((b & ~inner).sum())


@pytest.mark.parametrize("shape", [(2, 2, 2), (3, 5, 3), (2, 3, 4), (7, 6, 5), (9, 10, 33), (5, 40, 64), (21, 19, 130), (9, 8, 32), (17, 3, 31),
                                   (3, 4, 511), (3, 2, 529), (2, 5, 1100)])
@pytest.mark.parametrize("offset", [0, 1, 2, 7, 8, 13])
@pytest.mark.parametrize("p", [0.3, 0.97])
def test_volume_counts(gpu_ctx, shape, offset, p):
    import torch

    rng = np.random.default_rng(sum(shape) + offset)
    bone = (rng.random(shape) < 0.6).astype(np.uint8) * np.uint8(255)
    roi = (rng.random(shape) < p).astype(np.uint8)
    bone.flat[0] = roi.flat[0] = 1

    def on_gpu(a):  # at a byte offset from an aligned address
        t = torch.zeros(a.size + 32, dtype=torch.uint8, device="cuda")
        t[offset:offset + a.size] = torch.from_numpy(a.reshape(-1)).cuda()
        return t[offset:offset + a.size].view(a.shape)

    m = volume_metrics(on_gpu(bone), on_gpu(roi), 1.0, ctx=gpu_ctx)
    assert (m.bone_voxels, m.roi_voxels, m.boundary_bone_voxels) == counts(bone, roi)
