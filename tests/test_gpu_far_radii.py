"""Local thickness beyond the separable fill's radius (127 voxels): the 16-bit
distance transform's lines beyond 65 voxels are computed once in 32 bits, and
the tile fill takes them and the others as they are.  Against the oracle, bit
for bit."""

import numpy as np
import pytest

import oracle as O
from bone_morphometry_gb300 import (BoneMorphometryError, Phase, _lib, analyze_thickness,
                                    euclidean_distance_transform_squared, local_thickness)
from refstats import assert_reference_stats

pytestmark = pytest.mark.gpu


def sites(shape, points):
    vol = np.ones(shape, np.uint8)
    for p in points:
        vol[p] = 0
    return vol


CASES = [
    # every line along z flagged, some, and lines past a block's planes
    ("all-lines", sites((130, 9, 17), [(0, 0, 0)])),
    ("some-lines", sites((20, 20, 300), [(10, 10, x) for x in range(0, 120, 4)])),
    ("two-blocks", sites((70, 5, 280), [(69, 4, 0), (3, 0, 20)])),
    ("short", sites((2, 3, 200), [(0, 0, 0)])),
]


@pytest.mark.parametrize("name,vol", CASES, ids=[c[0] for c in CASES])
def test_far_radii_bitwise(gpu_ctx, name, vol):
    ref = O.local_thickness(vol, O.FOREGROUND)
    assert int(ref.edt.max()) > 127 * 127
    gpu_ctx.profile(True)
    got, sq = local_thickness(vol, Phase.FOREGROUND, ctx=gpu_ctx, return_squared=True)
    times = gpu_ctx.kernel_times()
    gpu_ctx.profile(False)
    assert np.array_equal(sq, ref.propagated)
    assert np.array_equal(got.view(np.uint32), ref.thickness.view(np.uint32))
    # x passes of 16 and of 32 bits, and no third
    assert times["edt_x"][0] == 2


@pytest.mark.parametrize("concurrent", [True, False])
def test_far_phase_beside_a_near_one(gpu_ctx, concurrent):
    bone = sites((20, 20, 300), [(10, 10, x) for x in range(0, 120, 4)])
    roi = np.ones_like(bone)
    gpu_ctx.set_concurrent_phases(concurrent)
    try:
        res = analyze_thickness(bone, roi, 3.0, ctx=gpu_ctx, return_maps=True)
    finally:
        gpu_ctx.set_concurrent_phases(True)
    for sel, got, gmap in ((True, res.thickness, res.thickness_map), (False, res.spacing, res.spacing_map)):
        ref = O.local_thickness(O.phase_inside(bone, roi, sel), O.FOREGROUND)
        assert np.array_equal(gmap.view(np.uint32), ref.thickness.view(np.uint32))
        assert_reference_stats(got, ref.thickness, 3.0)


@pytest.mark.parametrize("call", [local_thickness, euclidean_distance_transform_squared])
def test_all_selected_is_refused_after_one_transform(gpu_ctx, call):
    vol = np.ones((20, 30, 40), np.uint8)
    before = gpu_ctx.launches
    with pytest.raises(BoneMorphometryError) as e:
        call(vol, Phase.FOREGROUND, ctx=gpu_ctx)
    assert e.value.status == _lib.BM_ERR_ALL_SELECTED
    assert gpu_ctx.launches - before == 3  # x, y and z in 16 bits
