"""Batch prediction against a NumPy traversal that adds the leaves in forest
order in f32: host rows (feature-major on the device), device rows
(sample-major) and served rows, at the edges of the row tiles, of the
features staged per block and of the threshold search, must agree bit for bit.
"""
import ctypes

import numpy as np
import pytest

import boosters_b200 as bst
from boosters_b200 import _native

pytestmark = pytest.mark.gpu


def random_tree(rng, depth, pools, cat_feats, group=0):
    n = 2 ** (depth + 1) - 1
    level = np.floor(np.log2(np.arange(1, n + 1))).astype(int)
    leaf = (level == depth) | ((level >= 1) & (rng.random(n) < 0.1))
    feat = rng.integers(0, len(pools), n)
    cat = np.isin(feat, cat_feats) & ~leaf
    thr = np.array([rng.choice(pools[f]) for f in feat], np.float32)
    i = np.arange(n)
    return {"group": group, "split_index": np.where(leaf, 0, feat), "threshold": np.where(leaf | cat, 0, thr),
            "left": np.where(leaf, 0, np.minimum(2 * i + 1, n - 1)),
            "right": np.where(leaf, 0, np.minimum(2 * i + 2, n - 1)),
            "default_left": rng.integers(0, 2, n), "is_leaf": leaf.astype(np.uint8),
            "leaf_value": np.where(leaf, rng.standard_normal(n), 0).astype(np.float32),
            "split_type": cat.astype(np.uint8), "seg_start": np.where(cat, i, 0), "seg_size": cat.astype(np.uint32),
            "cat_words": rng.integers(0, 2 ** 32, n, dtype=np.uint64).astype(np.uint32)}


def walk(trees, x, n_groups, base):
    """x sample-major; f32 sums in forest order."""
    out = np.repeat(np.asarray(base, np.float32)[:, None], x.shape[0], 1)
    rows = np.arange(x.shape[0])
    for t in trees:
        node = np.zeros(x.shape[0], int)
        for _ in range(16):
            v = x[rows, t["split_index"][node]]
            with np.errstate(invalid="ignore"):
                left = v < t["threshold"][node]
                c = np.where(np.isnan(v) | (v <= 0), 0, np.minimum(v, 4e9)).astype(np.uint64)
            word = t["cat_words"][t["seg_start"][node]]
            right = (c < 32) & (((word >> (c % 32).astype(np.uint32)) & 1) == 1)
            left = np.where(t["split_type"][node] == 1, ~right, left)
            left = np.where(np.isnan(v), t["default_left"][node] == 1, left)
            node = np.where(t["is_leaf"][node] == 1, node, np.where(left, t["left"][node], t["right"][node]))
        out[t["group"]] += t["leaf_value"][node]
    return out


def check(trees, x, n_groups=1, base=(0.25,), server=True):
    import torch
    m = bst.GBDTModel.from_trees(x.shape[1], trees, bst.Objective.squared(), base)
    want = walk(trees, x, n_groups, base)
    np.testing.assert_array_equal(m.predict_group_major(bst.Dataset(x), raw=True), want)
    dx = torch.from_numpy(x).cuda()
    out = torch.empty((n_groups, x.shape[0]), device="cuda")
    _native.check(_native.lib.bst_gbdt_predict_device(
        m._h, ctypes.c_void_p(dx.data_ptr()), x.shape[0], x.shape[1], 1, ctypes.c_void_p(out.data_ptr()),
        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    np.testing.assert_array_equal(out.cpu().numpy(), want)
    if server:
        s = bst.PredictionServer(m, raw=True)
        try:
            np.testing.assert_array_equal(s.wait(s.submit(x)), want)
        finally:
            s.close()


def rows_of(rng, n, F, cat_feats=()):
    x = rng.standard_normal((n, F)).astype(np.float32)
    x[rng.random((n, F)) < 0.05] = np.nan
    x[rng.random((n, F)) < 0.01] = np.inf
    x[rng.random((n, F)) < 0.01] = -np.inf
    x[rng.random((n, F)) < 0.02] = 0.0
    for f in cat_feats:
        x[:, f] = rng.integers(-2, 40, n)
    return x


# rows: one, a warp's edge, the row groups' and tiles' edges, more than one
# wave of small tiles; features: one, around the staged eight; thresholds per
# feature: the search trees' edges and past the staged 255
@pytest.mark.parametrize("n,F,n_thr,depth,T", [
    (1, 1, 1, 1, 1), (31, 7, 15, 3, 5), (128, 8, 16, 4, 16), (129, 9, 17, 8, 17), (1000, 17, 31, 6, 40),
    (1025, 100, 127, 8, 33), (4097, 13, 240, 8, 70), (300, 3, 255, 8, 400), (300, 3, 256, 8, 400),
    (2000, 2, 700, 8, 300), (19_000, 5, 63, 5, 20), (40_000, 6, 200, 8, 12)])
def test_rows_features_thresholds(n, F, n_thr, depth, T):
    rng = np.random.default_rng(n * 131 + F)
    pools = [np.sort(np.concatenate([rng.standard_normal(n_thr - 1), [0.0]])).astype(np.float32) for _ in range(F)]
    trees = [random_tree(rng, depth, pools, []) for _ in range(T)]
    check(trees, rows_of(rng, n, F))


@pytest.mark.parametrize("n", [5, 700, 20_000])
def test_groups_and_categories(n):
    rng = np.random.default_rng(n)
    F, cats = 11, [2, 7]
    pools = [rng.standard_normal(20).astype(np.float32) for _ in range(F)]
    trees = [random_tree(rng, 6, pools, cats, group=i % 3) for i in range(31)]
    check(trees, rows_of(rng, n, F, cats), 3, (0.5, -1.0, 0.0))


def test_trees_too_deep_for_the_tiles():
    rng = np.random.default_rng(3)
    pools = [rng.standard_normal(50).astype(np.float32) for _ in range(4)]
    trees = [random_tree(rng, 10, pools, []) for _ in range(3)]
    check(trees, rows_of(rng, 500, 4))
