"""Host arrays reach the device the same through every form of the copy: pinned
(one asynchronous copy), pageable below the staging limit (the driver's copy)
and staged by 2 to 6 threads, at the sizes where the form changes and at sizes
that are no multiple of a block."""
import numpy as np
import pytest

import boosters_b200 as bst

pytestmark = pytest.mark.gpu

F = 7
TREE = {"group": 0, "split_index": np.array([F - 1, 0, 3, 0, 0, 0, 0]), "threshold": np.zeros(7, np.float32),
        "left": np.array([1, 3, 5, 0, 0, 0, 0]), "right": np.array([2, 4, 6, 0, 0, 0, 0]),
        "default_left": np.zeros(7, int), "is_leaf": np.array([0, 0, 0, 1, 1, 1, 1], np.uint8),
        "leaf_value": np.array([0, 0, 0, 1, 2, 4, 8], np.float32)}


@pytest.mark.parametrize("mib", [8, 16, 32, 48, 96])
@pytest.mark.parametrize("off", [-1, 0, 1])
def test_pageable_and_pinned_rows_agree(mib, off):
    import torch
    n = (mib << 20) // (4 * F) + off
    x = torch.randn((F, n), generator=torch.Generator().manual_seed(mib), dtype=torch.float32)
    m = bst.GBDTModel.from_trees(F, [TREE], bst.Objective.squared(), (0.0,))
    got = m.predict_group_major(bst.Dataset.from_feature_major(x.numpy()), raw=True)
    want = m.predict_group_major(bst.Dataset.from_feature_major(x.pin_memory().numpy()), raw=True)
    np.testing.assert_array_equal(got, want)
    a, b, c = x[F - 1].numpy() < 0, x[0].numpy() < 0, x[3].numpy() < 0
    np.testing.assert_array_equal(got[0], np.where(a, np.where(b, 1, 2), np.where(c, 4, 8)).astype(np.float32))
