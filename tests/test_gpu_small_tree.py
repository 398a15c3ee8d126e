"""Trees grown in one cooperative launch (small training sets) against the
level kernels, which a launch-shape cache file selects: nodes, sums, gains,
leaf values, row leaves and predictions must agree bit for bit, in every
gradient precision, with missing values, categories, sampling and weights, at
the sizes where the launch changes shape."""
import numpy as np
import pytest

import boosters_b200 as bst

pytestmark = pytest.mark.gpu


def both(tmp_path, ds, n, record=True, **kw):
    m = bst.GBDTModel.train(ds, bst.GBDTConfig(**kw), record_leaves=record)
    ref = bst.GBDTModel.train(ds, bst.GBDTConfig(autotune_cache=tmp_path / "shape.txt", **kw), record_leaves=record)
    assert m.tune_info.startswith("one launch per tree")
    assert not ref.tune_info.startswith("one launch")
    assert m.n_trees == ref.n_trees
    for i in range(m.n_trees):
        a, b = m.tree(i), ref.tree(i)
        for k in a:
            np.testing.assert_array_equal(a[k], b[k], err_msg=f"tree {i} {k}")
        if record:
            np.testing.assert_array_equal(m.tree_row_leaves(i, n), ref.tree_row_leaves(i, n))
    np.testing.assert_array_equal(m.train_predictions(), ref.train_predictions())
    return m


# rows below one per block, at warp and block edges, near the largest taken for
# few and for many columns; columns below, at and above one per SM; depths 1 to 8
@pytest.mark.parametrize("n,F,depth", [(40, 1, 1), (147, 3, 2), (149, 5, 3), (513, 33, 6), (2049, 148, 5),
                                       (3001, 150, 8), (5000, 100, 6), (27_900, 12, 7), (51_900, 80, 6)])
@pytest.mark.parametrize("precision", ["fp32", "q16", "q8"])
def test_sizes(tmp_path, n, F, depth, precision):
    x, y = bst.synth.regression(n, F, n_informative=min(F, 10), seed=n)
    ds = bst.Dataset.from_feature_major(x, y)
    both(tmp_path, ds, n, objective=bst.Objective.squared(), n_estimators=4, max_depth=depth, learning_rate=0.3,
         precision=precision)


# past one 16-bit-sum limit (q16: 65,536 rows)
@pytest.mark.parametrize("precision", ["q16", "q8"])
def test_most_rows(tmp_path, precision):
    x, y = bst.synth.regression(66_001, 80, n_informative=10, seed=7)
    ds = bst.Dataset.from_feature_major(x, y)
    both(tmp_path, ds, 66_001, objective=bst.Objective.squared(), n_estimators=4, max_depth=7, learning_rate=0.3,
         precision=precision)


@pytest.mark.parametrize("precision", ["fp32", "q8"])
@pytest.mark.parametrize("sampling", [{}, {"subsample": 0.7}, {"colsample_bytree": 0.5, "colsample_bylevel": 0.7},
                                      {"goss_top_rate": 0.2, "goss_other_rate": 0.2}])
def test_missing_values_and_sampling(tmp_path, precision, sampling):
    x, y = bst.synth.binary(9000, 30, n_nan_cols=9, seed=5)
    w = np.random.default_rng(1).uniform(0.1, 2.0, 9000).astype(np.float32)
    ds = bst.Dataset.from_feature_major(x, y, weights=w)
    both(tmp_path, ds, 9000, objective=bst.Objective.logistic(), n_estimators=6, max_depth=6, learning_rate=0.5,
         min_child_weight=3.0, min_gain_to_split=0.01, precision=precision, **sampling)


@pytest.mark.parametrize("precision", ["fp32", "q8"])
def test_categories_and_classes(tmp_path, precision):
    x, y = bst.synth.multiclass(7000, n_numeric=8, n_categorical=5, n_classes=4, seed=3)
    ds = bst.Dataset.from_feature_major(x, y, categorical_features=list(range(8, 13)))
    both(tmp_path, ds, 7000, objective=bst.Objective.softmax(4), n_estimators=3, max_depth=6, learning_rate=0.3,
         precision=precision)


def test_few_valued_and_many_binned_columns(tmp_path):
    rng = np.random.default_rng(8)
    n = 6000
    x = np.stack([rng.integers(0, k, n) for k in (2, 3, 17)] + [rng.standard_normal(n)] * 2).astype(np.float32)
    y = (x[0] * x[3] + np.sin(5 * x[2]) + 0.1 * rng.standard_normal(n)).astype(np.float32)
    ds = bst.Dataset.from_feature_major(x, y)
    both(tmp_path, ds, n, objective=bst.Objective.squared(), n_estimators=4, max_depth=7, learning_rate=0.3,
         max_bins=1500)


def test_no_split_and_early_leaves(tmp_path):
    rng = np.random.default_rng(9)
    x = rng.standard_normal((4, 300)).astype(np.float32)
    flat = bst.Dataset.from_feature_major(x, np.ones(300, np.float32))
    m = both(tmp_path, flat, 300, objective=bst.Objective.squared(), n_estimators=2, max_depth=4)
    assert all(len(m.tree(i)["is_leaf"]) == 1 for i in range(2))
    y = (x[0] > 1.2).astype(np.float32)
    both(tmp_path, bst.Dataset.from_feature_major(x, y), 300, objective=bst.Objective.logistic(), n_estimators=5,
         max_depth=8, min_samples_leaf=20)
