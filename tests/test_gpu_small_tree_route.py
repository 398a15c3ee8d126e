"""Which route a training set takes, one launch a tree or the level kernels: by
its rows, columns, depth, precision and the categories of its columns, on both
sides of the line."""
import numpy as np
import pytest

import boosters_b200 as bst

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,F,depth,precision,categories,one_launch", [
    (27_000, 12, 7, "fp32", 0, True), (27_000, 12, 8, "fp32", 0, False), (15_000, 12, 8, "fp32", 0, True),
    (51_000, 100, 6, "fp32", 0, True), (51_000, 100, 8, "fp32", 0, False), (65_000, 74, 6, "q16", 0, True),
    (66_000, 74, 8, "q16", 0, False), (69_000, 100, 4, "q8", 0, True), (69_000, 100, 8, "q8", 0, False),
    (13_000, 200, 6, "fp32", 0, True), (13_000, 200, 8, "fp32", 0, False), (9_000, 300, 8, "q8", 0, False),
    (20_000, 12, 6, "fp32", 20, True), (20_000, 12, 6, "fp32", 200, False), (20_000, 12, 8, "q8", 64, False),
    (4_000, 12, 6, "q8", 200, True)])
def test_route(n, F, depth, precision, categories, one_launch):
    rng = np.random.default_rng(n)
    x = rng.standard_normal((F, n)).astype(np.float32)
    cats = [F - 1] if categories else []
    if cats:
        x[-1] = np.arange(n) % categories
    y = (x[0] + 0.3 * rng.standard_normal(n)).astype(np.float32)
    m = bst.GBDTModel.train(bst.Dataset.from_feature_major(x, y, categorical_features=cats),
                            bst.GBDTConfig(n_estimators=1, max_depth=depth, precision=precision))
    assert m.tune_info.startswith("one launch per tree") == one_launch, m.tune_info
