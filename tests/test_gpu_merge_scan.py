"""The split search that merges the row segments' partial histograms itself,
against the host-driven levels (a merge kernel, then the search): trees agree
bit for bit for every number of warps a column gets (few and many columns,
shallow levels and ones of more than 256 nodes), with columns of the general
tiles (more than 264 bins), categories, missing values, sampling, and nodes
merged apart (more than 128 segments)."""
import numpy as np
import pytest

import boosters_b200 as bst

pytestmark = pytest.mark.gpu


def same(tmp_path, ds, **kw):
    a = bst.GBDTModel.train(ds, bst.GBDTConfig(autotune_cache=tmp_path / "shape.txt", **kw))
    b = bst.GBDTModel.train(ds, bst.GBDTConfig(batched=False, **kw))
    assert not a.tune_info.startswith("one launch")
    assert a.n_trees == b.n_trees
    for i in range(a.n_trees):
        ta, tb = a.tree(i), b.tree(i)
        for k in ta:
            np.testing.assert_array_equal(ta[k], tb[k], err_msg=f"tree {i} {k}")
    np.testing.assert_array_equal(a.train_predictions(), b.train_predictions())


@pytest.mark.parametrize("precision", ["fp32", "q16", "q8"])
@pytest.mark.parametrize("n,F,depth", [(3000, 1, 1), (20_000, 5, 8), (60_000, 75, 7), (9_000, 310, 5),
                                       (40_000, 6, 11)])
def test_columns_and_levels(tmp_path, precision, n, F, depth):
    x, y = bst.synth.binary(n, F, n_nan_cols=F // 3, seed=F)
    ds = bst.Dataset.from_feature_major(x, y)
    same(tmp_path, ds, objective=bst.Objective.logistic(), n_estimators=3, max_depth=depth, learning_rate=0.4,
         precision=precision)


@pytest.mark.parametrize("precision", ["fp32", "q8"])
@pytest.mark.parametrize("growth", ["depthwise", "leafwise"])
def test_wide_columns_categories_sampling(tmp_path, precision, growth):
    n = 30_000
    x, y = bst.synth.multiclass(n, n_numeric=9, n_categorical=4, n_classes=3, seed=4)
    kw = dict(growth_strategy=bst.GrowthStrategy.Leafwise, n_leaves=40) if growth == "leafwise" else dict(max_depth=6)
    for bins in (256, 700):  # 700: the numeric columns go to general tiles
        ds = bst.Dataset.from_feature_major(x, y, categorical_features=[9, 10, 11, 12])
        same(tmp_path, ds, objective=bst.Objective.softmax(3), n_estimators=2, learning_rate=0.3, max_bins=bins,
             precision=precision, colsample_bytree=0.8, subsample=0.8, **kw)


# fp32 segments hold 4096 rows: the root alone above 128 of them, then the
# levels too
@pytest.mark.parametrize("n", [560_000, 1_100_000])
@pytest.mark.parametrize("growth", ["depthwise", "leafwise"])
def test_nodes_of_many_segments(tmp_path, growth, n):
    x, y = bst.synth.regression(n, 4, n_informative=4, seed=9)
    kw = dict(growth_strategy=bst.GrowthStrategy.Leafwise, n_leaves=12) if growth == "leafwise" else dict(max_depth=4)
    ds = bst.Dataset.from_feature_major(x, y)
    same(tmp_path, ds, objective=bst.Objective.squared(), n_estimators=2, learning_rate=0.3, precision="fp32", **kw)
