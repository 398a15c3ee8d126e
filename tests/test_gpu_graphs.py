"""cuda_graph chooses how a tree's kernels are launched, one by one or as one
captured graph; trees, predictions and the phase timers agree either way."""
import numpy as np
import pytest

import boosters_b200 as bst

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("growth", ["depthwise", "leafwise"])
@pytest.mark.parametrize("extra", [{}, {"subsample": 0.7, "colsample_bytree": 0.6}, {"phase_timings": True}])
def test_graphs_and_plain_launches_agree(growth, extra):
    n = 80_000
    x, y = bst.synth.multiclass(n, n_numeric=10, n_categorical=3, n_classes=3, seed=2)
    ds = bst.Dataset.from_feature_major(x, y, categorical_features=[10, 11, 12])
    kw = dict(objective=bst.Objective.softmax(3), n_estimators=6, learning_rate=0.3, precision="q8", **extra)
    if growth == "leafwise":
        kw.update(growth_strategy=bst.GrowthStrategy.Leafwise, n_leaves=40)
    a, b = (bst.GBDTModel.train(ds, bst.GBDTConfig(cuda_graph=g, **kw)) for g in (False, True))
    assert a.n_trees == b.n_trees == 18
    for i in range(18):
        ta, tb = a.tree(i), b.tree(i)
        for k in ta:
            np.testing.assert_array_equal(ta[k], tb[k], err_msg=f"tree {i} {k}")
    np.testing.assert_array_equal(a.train_predictions(), b.train_predictions())
    if "phase_timings" in extra:
        for m in (a, b):
            t = m.train_timings()
            assert all(t[k] > 0 for k in ("gradients", "histograms", "split_scan", "partition", "leaf_update")), t
            assert sum(v for k, v in t.items() if k not in ("binning", "total")) <= 1.2 * t["total"], t
