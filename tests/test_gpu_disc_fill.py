"""The separable sphere fill against the oracle, at the edges of its patches
(32 x 8 columns), tiles (64 x 32) and plane runs (32), at small and large radii
and beyond its radius limit.  The maps are whole numbers or the reference's own
f32 arithmetic, so the comparison is bit for bit."""

import numpy as np
import pytest

import oracle as O
from bone_morphometry_gb300 import Phase, local_thickness

pytestmark = pytest.mark.gpu


def blobs(shape, sigma, frac, seed):
    from scipy.ndimage import gaussian_filter

    f = gaussian_filter(np.random.default_rng(seed).standard_normal(shape).astype(np.float32), sigma)
    return (f > np.quantile(f, 1 - frac)).astype(np.uint8)


def one_site(shape, at):
    vol = np.ones(shape, np.uint8)
    vol[at] = 0
    return vol


CASES = [
    # (d, h, w) below, at and past the patch, tile and plane-run edges
    ("tiny", lambda: blobs((2, 2, 2), 0.5, 0.5, 1)),
    ("edges-1", lambda: blobs((31, 31, 63), 1.5, 0.6, 2)),
    ("edges", lambda: blobs((32, 32, 64), 1.5, 0.6, 3)),
    ("edges+1", lambda: blobs((33, 33, 65), 1.5, 0.6, 4)),
    ("patch-rows", lambda: blobs((40, 9, 97), 2.0, 0.7, 5)),
    ("thin", lambda: blobs((3, 70, 130), 2.0, 0.5, 6)),
    ("noise", lambda: (np.random.default_rng(7).random((37, 41, 70)) < 0.7).astype(np.uint8)),
    ("sparse-sites", lambda: (np.random.default_rng(8).random((50, 60, 70)) < 0.9995).astype(np.uint8)),
    ("thick", lambda: blobs((72, 80, 100), 9.0, 0.8, 9)),
    # long lists: distances that rise along a line
    ("ramp", lambda: one_site((61, 20, 20), (0, 0, 0))),
    ("limit", lambda: one_site((126, 8, 16), (0, 0, 7))),     # largest squared radius 15738: below 127^2
    ("beyond", lambda: one_site((128, 8, 16), (0, 0, 7))),    # 16242: the tile fill
    ("overfull", lambda: (np.random.default_rng(10).random((40, 40, 70)) < 0.5).astype(np.uint8)),
]


@pytest.mark.parametrize("name,make", CASES, ids=[c[0] for c in CASES])
@pytest.mark.parametrize("phase", [Phase.FOREGROUND, Phase.BACKGROUND])
def test_separable_fill_bitwise(gpu_ctx, name, make, phase):
    vol = make()
    if phase == Phase.BACKGROUND:
        vol = 1 - vol
    if not (vol == 0).any() or not (vol != 0).any():
        vol.flat[0] = 1 - vol.flat[0]
    ref = O.local_thickness(vol, int(phase))
    got, sq = local_thickness(vol, phase, ctx=gpu_ctx, return_squared=True)
    assert np.array_equal(sq, ref.propagated)
    assert np.array_equal(got.view(np.uint32), ref.thickness.view(np.uint32))


@pytest.mark.parametrize("d,w", [(7, 70), (8, 70), (9, 70), (17, 33), (31, 1300), (32, 1300), (33, 1300), (65, 1000)])
def test_plane_runs_bitwise(gpu_ctx, d, w):
    """Runs of 8 planes (narrow volumes) and of 32 (wide ones), at their edges."""
    vol = blobs((d, 17, w), 2.0, 0.6, d + w)
    ref = O.local_thickness(vol, 0)
    got, sq = local_thickness(vol, Phase.FOREGROUND, ctx=gpu_ctx, return_squared=True)
    assert np.array_equal(sq, ref.propagated)
    assert np.array_equal(got.view(np.uint32), ref.thickness.view(np.uint32))


def test_lists_that_outgrow_their_pool():
    """Balls that overlap at random want more list entries than their radius
    suggests: the first call fills again in a larger pool, the second at once."""
    from bone_morphometry_gb300 import Context

    ctx = Context(0)
    vol = (np.random.default_rng(11).random((90, 100, 130)) < 0.9995).astype(np.uint8)
    ref = O.local_thickness(vol, 0)
    launches = []
    for _ in range(2):
        before = ctx.launches
        got, sq = local_thickness(vol, Phase.FOREGROUND, ctx=ctx, return_squared=True)
        launches.append(ctx.launches - before)
        assert np.array_equal(sq, ref.propagated)
        assert np.array_equal(got.view(np.uint32), ref.thickness.view(np.uint32))
    ctx.close()
    # 3 launches make the tables of a new context, 5 fill again
    assert launches[0] == launches[1] + 3 + 5
