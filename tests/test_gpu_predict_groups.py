"""Forests of several outputs and categorical splits large enough for a small
batch to split their trees over blocks, at one and several staged chunks of
trees an output and on both sides of the limit of leaf values, against the NumPy
traversal; and served rows against the node list, which a tree too deep for the
tiles (its leaves zero) selects."""
import numpy as np
import pytest

import boosters_b200 as bst
from test_gpu_predict_paths import check, random_tree, rows_of

pytestmark = pytest.mark.gpu

F, CATS = 11, [2, 7]


def forest(seed, n_trees, groups, depth=6):
    rng = np.random.default_rng(seed)
    pools = [rng.standard_normal(20).astype(np.float32) for _ in range(F)]
    return [random_tree(rng, depth, pools, CATS, group=i % groups) for i in range(n_trees)]


# 96 trees: the least that are split; 801: 267 an output, more than one chunk;
# 15,600 x 801 rows of 128: just under the limit of leaf values, 16,000 past it
@pytest.mark.parametrize("n_trees,n", [(95, 129), (96, 1), (97, 129), (100, 5000), (801, 1), (801, 129),
                                       (801, 15_600), (801, 16_000)])
def test_groups_and_categories_of_split_forests(n_trees, n):
    rng = np.random.default_rng(n + n_trees)
    check(forest(n_trees, n_trees, 3), rows_of(rng, n, F, CATS), 3, (0.5, -1.0, 0.0))


@pytest.mark.parametrize("n", [1, 700, 40_000])
def test_served_rows_match_the_node_list(n):
    rng = np.random.default_rng(n)
    trees, x = forest(5, 120, 2, depth=8), rows_of(rng, n, F, CATS)
    deep = random_tree(rng, 9, [np.zeros(3, np.float32)] * F, [])
    deep["leaf_value"] = np.zeros_like(deep["leaf_value"])
    m, node_list = (bst.GBDTModel.from_trees(F, t, bst.Objective.squared(), (0.25, -0.5)) for t in (trees, trees + [deep]))
    want = node_list.predict_group_major(bst.Dataset(x), raw=True)
    np.testing.assert_array_equal(m.predict_group_major(bst.Dataset(x), raw=True), want)
    srv = bst.PredictionServer(m, raw=True)
    try:
        np.testing.assert_array_equal(srv.wait(srv.submit(x)), want)
    finally:
        srv.close()
