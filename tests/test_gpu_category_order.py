"""The order of a column's categories in the split search (by gradient ratio,
equal ones by category) at the warp and word edges of its number, with equal
ratios and categories without rows, in every form that searches columns: the
host-driven levels, the level kernels and the one launch a tree, against the
oracle."""
import numpy as np
import pytest

import boosters_b200 as bst
import oracle_bridge as ob
from test_gpu_parity import compare_trees

pytestmark = pytest.mark.gpu

COUNTS = [2, 4, 5, 31, 32, 33, 63, 64, 65, 128, 129, 192, 255, 256]


@pytest.mark.parametrize("form", ["host", "levels", "one launch"])
@pytest.mark.parametrize("k", COUNTS)
def test_order(form, k):
    n = k * max(20, (60_000 if form == "levels" else 4_000) // k + 1)
    rng = np.random.default_rng(k)
    cat = np.arange(n) % k
    step = rng.permutation(k)[: k // 2 + 1].astype(np.float32)
    y = (step[cat // 2] / 8 + (np.arange(n) // k % 4) / 2).astype(np.float32)  # pairs of categories tie
    other = rng.integers(0, max(2, k // 3), n)
    other[other == 1] = 0  # a category without rows below the largest
    x = np.stack([cat, other, rng.standard_normal(n)]).astype(np.float32)
    cfg = bst.GBDTConfig(objective=bst.Objective.squared(), n_estimators=2, max_depth=4, learning_rate=0.5,
                         batched=form != "host")
    ds = bst.Dataset.from_feature_major(x, y, categorical_features=[0, 1])
    gm = bst.GBDTModel.train(ds, cfg, n_threads=1, record_leaves=True)
    assert gm.tune_info.startswith("one launch") == (form == "one launch")
    compare_trees(gm, ob.OracleModel(x, y, cfg.to_c(), n_threads=1, categorical=[0, 1]), n)
