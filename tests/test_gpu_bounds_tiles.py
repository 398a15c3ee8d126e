"""Numeric bin bounds (a block's radix sort) at the edges of its 8192-key tiles
and for keys whose digits are skewed (whole numbers, one value, few high
bytes) or not (random bits), against the oracle, bit for bit."""
import numpy as np
import pytest

import boosters_b200 as bst
import oracle_bridge as ob

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 33, 511, 8191, 8192, 8193, 24_577, 200_000, 200_003])
def test_bounds_match_the_oracle(n):
    rng = np.random.default_rng(n)
    bits = rng.integers(0, 2**32, n, dtype=np.uint32).view(np.float32)  # infinities and NaN among them
    one = np.full(n, 3.0, np.float32)
    one[-1] = 2.5
    x = np.stack([
        np.where(np.isnan(bits), np.float32("nan"), bits).astype(np.float32),
        rng.integers(-3000, 3000, n).astype(np.float32),
        one,
        rng.normal(size=n).astype(np.float32),
        (1.0 + np.arange(n) * 2.0**-22).astype(np.float32)[::-1],
    ])
    cfg = bst.GBDTConfig(max_bins=255)
    got = bst.BinnedDataset(bst.Dataset.from_feature_major(np.ascontiguousarray(x)), cfg)
    want = ob.OracleBinned(x, cfg.to_c())
    assert got.n_columns == want.n_columns
    for c in range(got.n_columns):
        np.testing.assert_array_equal(got.column_bounds(c), want.column_bounds(c), err_msg=f"column {c}")
        np.testing.assert_array_equal(got.column_bins(c), want.column_bins(c), err_msg=f"column {c}")
