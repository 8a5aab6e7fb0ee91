"""Device memory: a server's worker stays within the estimate that admits its
requests, and volumes a few voxels wide within what their size asks for."""

from contextlib import closing

import numpy as np
import pytest

import oracle as O
from bone_morphometry_gb300 import Context, FeatureMode, Phase, analyze_thickness, local_thickness
from bone_morphometry_gb300.serving import Server, footprint_bytes

pytestmark = pytest.mark.gpu


def free_bytes():
    import torch

    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def two_halves(shape, spacing, seed):
    """Bone with marrow voxels about `spacing` apart, then marrow with bone voxels as far apart."""
    d, h, w = shape
    rng = np.random.default_rng(seed)
    vol = np.ones(shape, np.uint8)
    vol[d // 2:] = 0
    for z in range(spacing // 2, d, spacing):
        for y in range(spacing // 2, h, spacing):
            for x in range(spacing // 2, w, spacing):
                at = tuple(min(max(int(c + rng.integers(-6, 7)), 0), n - 1) for c, n in ((z, d), (y, h), (x, w)))
                vol[at] = 1 - vol[at]
    return vol


def test_requests_stay_within_their_footprint():
    """Large radii (list pools above a byte per voxel) in a cross-section just past
    a patch's edge (padded lists and rows), with and without quantiles."""
    shape = (3000, 129, 129)
    bone = two_halves(shape, 64, 21)
    roi = np.ones_like(bone)
    modes = (FeatureMode.CLASSIC, FeatureMode.STANDARD)
    with closing(Context(0)) as ctx:
        alone = [analyze_thickness(bone, roi, 10.0, feature_mode=m, ctx=ctx) for m in modes]
    before = free_bytes()
    with Server(workers=1, hbm_budget_bytes=200e9) as srv:
        for m, a in zip(modes, alone):
            r = srv.result(srv.submit(bone, roi, 10.0, feature_mode=m))
            assert r.status == 0 and r.footprint_bytes == footprint_bytes(shape)
            assert before - free_bytes() <= r.footprint_bytes
            for got, want in ((r.thickness, a.thickness), (r.spacing, a.spacing)):
                assert repr(got) == repr(want)


@pytest.mark.parametrize("w", [2, 3, 7, 8, 9, 17])
def test_narrow_volumes_bitwise(gpu_ctx, w):
    vol = (np.random.default_rng(w).random((60, 70, w)) < 0.97).astype(np.uint8)
    ref = O.local_thickness(vol, O.FOREGROUND)
    got, sq = local_thickness(vol, Phase.FOREGROUND, ctx=gpu_ctx, return_squared=True)
    assert np.array_equal(sq, ref.propagated)
    assert np.array_equal(got.view(np.uint32), ref.thickness.view(np.uint32))


def test_wide_thin_volume_takes_no_lists():
    """Two voxels wide: lists would take 200 bytes a voxel, 2.5 GB here."""
    shape = (2600, 2400, 2)
    vol = (np.random.default_rng(5).random(shape) < 0.9).astype(np.uint8)
    before = free_bytes()
    with closing(Context(0)) as ctx:
        got = local_thickness(vol, Phase.FOREGROUND, ctx=ctx)
        assert before - free_bytes() <= footprint_bytes(shape)
    assert np.array_equal(got.view(np.uint32), O.local_thickness(vol, O.FOREGROUND).thickness.view(np.uint32))


def test_a_worker_that_changes_between_fills():
    """One worker: the separable fill, the tile fill (radii above 127), the first again."""
    near = (np.random.default_rng(8).random((40, 50, 60)) < 0.9).astype(np.uint8)
    far = np.ones((20, 20, 300), np.uint8)
    far[10, 10, :120:4] = 0
    order = (near, far, near, far, near)
    with closing(Context(0)) as ctx:
        alone = [analyze_thickness(v, np.ones_like(v), 5.0, ctx=ctx) for v in order]
    with Server(workers=1, hbm_budget_bytes=20e9) as srv:
        for v, a in zip(order, alone):
            r = srv.result(srv.submit(v, np.ones_like(v), 5.0))
            assert r.status == 0
            assert repr(r.thickness) == repr(a.thickness) and repr(r.spacing) == repr(a.spacing)
