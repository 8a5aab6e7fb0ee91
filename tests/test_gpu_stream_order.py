"""Device-tensor calls run after the work on the caller's stream that produces their inputs."""

import numpy as np
import pytest

import oracle as O
from bone_morphometry_gb300 import euclidean_distance_transform_squared, serving
from bone_morphometry_gb300 import synthetic as S

pytestmark = pytest.mark.gpu

_BUSY_CYCLES = 40_000_000  # about 20 ms of a spinning kernel before the input is written


@pytest.mark.parametrize("side_stream", [False, True])
def test_input_written_just_before_the_call(gpu_ctx, side_stream):
    import torch

    rng = np.random.default_rng(3)
    vol = (rng.random((20, 24, 33)) < 0.8).astype(np.uint8)
    src = torch.from_numpy(vol).cuda()
    dst = torch.zeros_like(src)
    torch.cuda.synchronize()
    with torch.cuda.stream(torch.cuda.Stream() if side_stream else torch.cuda.default_stream()):
        torch.cuda._sleep(_BUSY_CYCLES)
        dst.copy_(src)
        out = euclidean_distance_transform_squared(dst, ctx=gpu_ctx)
    torch.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy().view(np.uint32), O.edt_sq(vol))


def test_batch_inputs_written_just_before_the_call(gpu_ctx):
    import torch

    sp = S.make_specimen((24, 40, 48), 2.0, 0.3, "cylinder", 18.0, 10.0, seed=9)
    bone, roi = torch.from_numpy(sp.bone).cuda(), torch.from_numpy(sp.roi).cuda()
    dst = torch.zeros_like(bone)
    torch.cuda.synchronize()
    torch.cuda._sleep(_BUSY_CYCLES)
    dst.copy_(bone)
    th, _, status = serving.batch_tbth_tbsp([serving.SpecimenInput(dst, roi, 10.0)], ctx=gpu_ctx)[0]
    ref = O.local_thickness(O.phase_inside(sp.bone, sp.roi, True), O.FOREGROUND).thickness
    assert status == 0 and th.mean == O.nonzero_stats(ref, 10.0).mean
