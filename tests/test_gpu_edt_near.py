"""The 16-bit distance passes against the oracle at the edges of their eights of
x, 64-column tiles, 128-row chunks and 64-row halos, around the largest distance
they hold (65 voxels) and beyond it, where the 32-bit passes compute the flagged
lines.  Squared distances are whole numbers: the comparison is exact."""

import numpy as np
import pytest

import oracle as O
from bone_morphometry_gb300 import Phase, local_thickness
from bone_morphometry_gb300 import euclidean_distance_transform_squared as edt

pytestmark = pytest.mark.gpu


def sites(shape, at):
    vol = np.ones(shape, np.uint8)
    for p in at:
        vol[p] = 0
    return vol


def noise(shape, p, seed):
    return (np.random.default_rng(seed).random(shape) < p).astype(np.uint8)


def near_and_far(shape, seed):  # most columns near a site, one corner far from any
    vol = noise(shape, 0.97, seed)
    vol[: shape[0] // 2, : shape[1] // 2, : shape[2] // 2] = 1
    return vol


CASES = [("noise-%d-%d-%d" % s, lambda s=s: noise(s, 0.96, sum(s)))
         for s in [(3, 5, 2), (4, 3, 7), (127, 9, 8), (128, 129, 9), (129, 127, 17), (5, 64, 63), (6, 65, 65),
                   (3, 4, 255), (4, 5, 256), (5, 6, 257), (260, 3, 31), (3, 260, 129), (2, 2, 1100)]]
# one site: the largest squared distance lies just below, at and above 65^2 along each axis
for n in (65, 66, 67, 130, 199, 257):
    CASES += [("x-%d" % n, lambda n=n: sites((3, 4, n), [(0, 0, 0)])),
              ("y-%d" % n, lambda n=n: sites((3, n, 5), [(2, 0, 4)])),
              ("z-%d" % n, lambda n=n: sites((n, 3, 4), [(n - 1, 2, 0)]))]
CASES += [
    ("diagonal", lambda: sites((50, 60, 70), [(0, 0, 0)])),
    ("two-far", lambda: sites((150, 140, 97), [(3, 5, 7), (149, 100, 90)])),
    ("part-far", lambda: near_and_far((160, 150, 140), 1)),
    ("part-far-odd", lambda: near_and_far((141, 153, 167), 2)),
    ("row-reach", lambda: sites((2, 2, 600), [(0, 0, 0), (0, 0, 400), (1, 1, 590)])),
]


@pytest.mark.parametrize("name,make", CASES, ids=[c[0] for c in CASES])
@pytest.mark.parametrize("phase", [Phase.FOREGROUND, Phase.BACKGROUND])
def test_edt_bitwise(gpu_ctx, name, make, phase):
    vol = make()
    if phase == Phase.BACKGROUND:
        vol = 1 - vol
    assert np.array_equal(edt(vol, phase, ctx=gpu_ctx), O.edt_sq(vol, int(phase)))


@pytest.mark.parametrize("w", [64, 112, 1040])
@pytest.mark.parametrize("tiles", [False, True])
def test_sites_outside_the_first_word(gpu_ctx, w, tiles):
    """No site in the first 32 of any 512 columns: both forms of the x pass count the others."""
    vol = noise((9, 11, w), 0.9, w)
    for x in range(0, w, 512):
        vol[:, :, x : x + 32] = 1
    gpu_ctx.set_fill_tile_rows(16 if tiles else 0)
    try:
        got = local_thickness(vol, Phase.FOREGROUND, ctx=gpu_ctx)
    finally:
        gpu_ctx.set_fill_tile_rows(0)
    assert np.array_equal(got.view(np.uint32), O.local_thickness(vol, 0).thickness.view(np.uint32))


@pytest.mark.parametrize("shape", [(5, 6, 15), (4, 9, 16), (7, 5, 17), (9, 7, 59), (5, 33, 60), (6, 4, 61), (33, 8, 119),
                                   (35, 5, 121), (70, 9, 31), (75, 71, 66), (131, 20, 15)])
def test_ridge_of_pairs_bitwise(gpu_ctx, shape):
    """Ridge map at the edges of its 60-voxel warps and padded rows; the last two
    shapes hold squared distances beyond 65^2 (16-bit map from flagged lines)."""
    vol = noise(shape, 0.9, sum(shape))
    if shape[0] > 70:
        vol[:] = 1
        vol[0, 0, shape[2] - 1] = 0
    got, sq = local_thickness(vol, Phase.FOREGROUND, ctx=gpu_ctx, return_squared=True)
    ref = O.local_thickness(vol, 0)
    assert np.array_equal(sq, ref.propagated)
    assert np.array_equal(got.view(np.uint32), ref.thickness.view(np.uint32))


@pytest.mark.parametrize("offset", [0, 1, 2, 3, 4, 8, 11, 12, 15])
@pytest.mark.parametrize("shape", [(2, 2, 2), (2, 3, 5), (3, 2, 15), (3, 5, 16), (2, 4, 17), (3, 3, 31), (2, 2, 33), (4, 3, 511), (3, 2, 529)])
def test_rows_at_any_address(gpu_ctx, shape, offset):
    """Rows that start at any byte: words that hang over either end of the volume."""
    import torch

    vol = noise(shape, 0.8, sum(shape))
    vol.flat[0] = 0
    vol.flat[-1] = 1
    t = torch.full((vol.size + 16,), 1, dtype=torch.uint8, device="cuda")
    t[offset : offset + vol.size] = torch.from_numpy(vol).cuda().flatten()
    view = t[offset : offset + vol.size].view(shape)
    got = edt(view, Phase.FOREGROUND, ctx=gpu_ctx)
    assert np.array_equal(got.cpu().numpy().view(np.uint32), O.edt_sq(vol, 0))
