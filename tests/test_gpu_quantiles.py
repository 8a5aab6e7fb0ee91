"""Order statistics and exact sums on values that stress the histograms (exact
results: compared for equality)."""

import numpy as np
import pytest

import oracle as O
from bone_morphometry_gb300 import nonzero_stats
from refstats import assert_reference_stats

pytestmark = pytest.mark.gpu


VALUES = {
    "constant": lambda r, n: np.full(n, 3.5, np.float32),
    "few distinct": lambda r, n: (2.0 * np.sqrt(r.integers(1, 9, n))).astype(np.float32),
    "one high bin": lambda r, n: (1.0 + r.random(n) / 256).astype(np.float32),
    "all exponents": lambda r, n: np.exp2(r.uniform(-148, 127, n)).astype(np.float32),
    "rising": lambda r, n: np.exp2(np.linspace(-60, 60, n)).astype(np.float32),
    "subnormal": lambda r, n: (r.integers(1, 1 << 20, n) * 1.4e-45).astype(np.float32),
}


@pytest.mark.parametrize("kind", VALUES)
@pytest.mark.parametrize("n", [1, 3, 4, 130, 100_003])
def test_order_statistics_and_exact_sums(gpu_ctx, kind, n):
    rng = np.random.default_rng(n)
    v = VALUES[kind](rng, n)
    if n > 4:
        v[rng.random(n) < 0.3] = 0
        v[rng.random(n) < 0.02] = [np.nan, np.inf, -2.0][n % 3]
    v[0] = max(v[0], np.float32(1e-44)) if v[0] == v[0] else np.float32(1.0)
    st = nonzero_stats(v, 1.0, True, ctx=gpu_ctx)
    med, p10, p25, p75, p90 = O.quantiles(v, 1.0, (0.5, 0.1, 0.25, 0.75, 0.9))
    assert (st.median, st.percentile_10, st.percentile_25, st.percentile_75, st.percentile_90) == (med, p10, p25, p75, p90)
    assert_reference_stats(st, v, 1.0)
