"""Calls whose device allocations fail part way, injected on the host
(Context.fail_allocation): they fall back or report BM_ERR_OOM, and the context
stays usable.  Maps bit for bit against the oracle."""

import numpy as np
import pytest

import oracle as O
from refstats import assert_reference_stats
from bone_morphometry_gb300 import BoneMorphometryError, Context, Phase, _lib, analyze_thickness, local_thickness

pytestmark = pytest.mark.gpu


@pytest.fixture
def ctx():
    c = Context(0)
    yield c
    c.close()


def random_balls(shape=(90, 100, 130), seed=11):
    """Balls that overlap at random: more list entries than their radius suggests."""
    return (np.random.default_rng(seed).random(shape) < 0.9995).astype(np.uint8)


def assert_maps(res, bone, roi, spacing):
    for sel, got, gmap in ((True, res.thickness, res.thickness_map), (False, res.spacing, res.spacing_map)):
        ref = O.local_thickness(O.phase_inside(bone, roi, sel), O.FOREGROUND)
        assert np.array_equal(gmap.view(np.uint32), ref.thickness.view(np.uint32))
        assert_reference_stats(got, ref.thickness, spacing)


@pytest.mark.parametrize("concurrent", [True, False])
def test_bone_phase_whose_pool_cannot_grow(ctx, concurrent):
    """The bone phase turns to the tile fill at its end, the marrow phase beside it does not."""
    bone = random_balls()
    roi = np.ones_like(bone)
    ctx.set_concurrent_phases(concurrent)
    ctx.fail_allocation("disc pool", 1)
    ctx.profile(True)
    res = analyze_thickness(bone, roi, 12.5, ctx=ctx, return_maps=True)
    times = ctx.kernel_times()
    ctx.profile(False)
    assert times["fill_rank"][0] > 0  # the tile fill ran
    assert_maps(res, bone, roi, 12.5)
    # the injection is spent: the lists again
    assert_maps(analyze_thickness(bone, roi, 12.5, ctx=ctx, return_maps=True), bone, roi, 12.5)


def assert_thickness(ctx, vol):
    ref = O.local_thickness(vol, O.FOREGROUND)
    got, sq = local_thickness(vol, Phase.FOREGROUND, ctx=ctx, return_squared=True)
    assert np.array_equal(sq, ref.propagated)
    assert np.array_equal(got.view(np.uint32), ref.thickness.view(np.uint32))


@pytest.mark.parametrize("what,skip", [("template table", 0), ("diameter table", 0), ("disc tables", 0),
                                       ("disc tables", 1)])
def test_tables_by_radius_after_a_failed_allocation(ctx, what, skip):
    """A context's first tables, and their growth: the call reports it and the next ones are exact."""
    rng = np.random.default_rng(3)
    small = (rng.random((20, 24, 40)) < 0.8).astype(np.uint8)
    large = np.ones((90, 12, 20), np.uint8)  # squared radii to 7921: the tables grow
    large[0, 0, 0] = 0
    for vol in (small, large):
        ctx.fail_allocation(what, skip)
        with pytest.raises(BoneMorphometryError) as e:
            local_thickness(vol, Phase.FOREGROUND, ctx=ctx)
        assert e.value.status == _lib.BM_ERR_OOM and what in str(e.value)
        if vol is large:
            assert_thickness(ctx, small)
        assert_thickness(ctx, vol)


LIST_BUFFERS = ["disc headers", "disc lists", "disc pool"]


@pytest.mark.parametrize("what", LIST_BUFFERS)
def test_no_memory_for_the_lists(ctx, what):
    """The first allocation of any of the lists' buffers fails: the tile fill."""
    vol = random_balls((40, 50, 70))
    ctx.fail_allocation(what)
    ctx.profile(True)
    assert_thickness(ctx, vol)
    assert ctx.kernel_times()["fill_rank"][0] > 0
    ctx.profile(True)
    assert_thickness(ctx, vol)  # the injection is spent: the lists
    assert ctx.kernel_times()["fill_rank"][0] == 0
    ctx.profile(False)


@pytest.mark.parametrize("shape", [(40, 50, 70), (90, 100, 130)])
def test_no_memory_for_one_phases_lists(ctx, shape):
    """The bone phase's pool only; phases launched in turns (below 2^20 voxels) or one after the other."""
    bone = random_balls(shape)
    roi = np.ones_like(bone)
    ctx.fail_allocation("disc pool")
    assert_maps(analyze_thickness(bone, roi, 7.0, ctx=ctx, return_maps=True), bone, roi, 7.0)
