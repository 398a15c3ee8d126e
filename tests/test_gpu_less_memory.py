"""Calls that fit the device memory only in their smaller form take it, with the
same results: leaf-wise growth without its speculative slots, under the
library's memory cap in a child process."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

TRAIN = r"""
import sys, hashlib
sys.path.insert(0, sys.argv[1])
import numpy as np
import boosters_b200 as bst
x, y = bst.synth.binary(20_000, 100, 0, seed=5)
ds = bst.Dataset.from_feature_major(x, y)
kw = dict(objective=bst.Objective.logistic(), n_estimators=2, n_leaves=512, precision="q8",
          growth_strategy=bst.GrowthStrategy.Leafwise)
val = bst.Dataset.from_feature_major(x[:, :5000].copy(), y[:5000].copy())

def fields(m):
    h = hashlib.sha256()
    for i in range(m.n_trees):
        t = m.tree(i)
        for k in ("split_index", "split_bin", "left", "right", "leaf_value", "gain"):
            h.update(np.ascontiguousarray(t[k]).tobytes())
    return h.hexdigest()

booster = bst.Booster(ds, bst.GBDTConfig(**kw))
booster.update(2)
out = [fields(booster.model())]
del booster
out.append(fields(bst.GBDTModel.train(ds, bst.GBDTConfig(**kw))))
out.append(fields(bst.GBDTModel.train(ds, bst.GBDTConfig(early_stopping_rounds=5, **kw), val_set=val)))
out.append(fields(bst.GBDTModel.grow_tree(ds, (0.5 - y).astype(np.float32), np.full(len(y), 0.25, np.float32),
                                          bst.GBDTConfig(**dict(kw, n_leaves=300)))))
print("trees", *out)
"""


def trees(limit):
    env = {k: v for k, v in os.environ.items() if k != "BST_DEVICE_MEMORY_LIMIT"}
    if limit:
        env["BST_DEVICE_MEMORY_LIMIT"] = str(limit << 20)
    r = subprocess.run([sys.executable, "-c", TRAIN, ROOT], capture_output=True, text=True, env=env, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    return next(ln for ln in r.stdout.split("\n") if ln.startswith("trees"))


# the buffers take about 690 MiB with the slots, 540 without
@pytest.mark.parametrize("limit", [560, 620])
def test_leafwise_without_speculation(limit):
    assert trees(limit) == trees(None)
