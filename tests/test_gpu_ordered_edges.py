"""The reference-order sums at the edges of chunks (256 values), blocks (8192) and
the two kernel shapes (2^22 values), at unaligned addresses, with ties, and with
more binade crossings than the walker prepares.  The sums are the reference's
own f64 results: compared for equality."""

import numpy as np
import pytest

import oracle as O
from bone_morphometry_gb300 import nonzero_stats

pytestmark = pytest.mark.gpu

KINDS = {
    "diameters": lambda r, n: np.where(r.random(n) < 0.4, 2.0 * np.sqrt(r.integers(1, 900, n)), 0.0).astype(np.float32),
    # whole numbers and halves: ties as soon as the sums pass 2^53 ulps of a half
    "ties": lambda r, n: (r.integers(1, 64, n) * 0.5 + 2.0 ** -20 * r.integers(0, 2, n)).astype(np.float32),
    "wide": lambda r, n: np.exp2(r.uniform(-20, 20, n)).astype(np.float32),
}


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n", [1, 255, 256, 257, 8191, 8192, 8193, 262_145, (1 << 22) - 1, 1 << 22, (1 << 22) + 77])
@pytest.mark.parametrize("offset", [0, 1])
def test_sums_at_the_edges(gpu_ctx, kind, n, offset):
    import torch

    v = KINDS[kind](np.random.default_rng(n), n)
    v[0] = 3.0
    t = torch.zeros(n + 4, dtype=torch.float32, device="cuda")
    t[offset:offset + n] = torch.from_numpy(v).cuda()
    st = nonzero_stats(t[offset:offset + n], 19.5, ctx=gpu_ctx)
    seq = O.nonzero_stats(v, 19.5)
    assert (st.count, st.sum, st.sum_of_squares) == (seq.count, seq.sum, seq.sum_sq)


def test_more_crossings_than_the_walker_prepares(gpu_ctx):
    v = np.exp2(np.linspace(-120, 60, 3_000_000)).astype(np.float32)  # the squares cross 360 binades
    st = nonzero_stats(v, 1.0, ctx=gpu_ctx)
    seq = O.nonzero_stats(v, 1.0)
    assert (st.count, st.sum, st.sum_of_squares) == (seq.count, seq.sum, seq.sum_sq)
