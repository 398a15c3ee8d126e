"""Calls that fit the device memory only in their smaller form take it, with the
same results: leaf-wise growth without its speculative slots, under the
library's memory cap, and prediction of device rows without room to split the
trees, with the rest of the device held; each in a child process."""
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


PREDICT = r"""
import sys, ctypes
sys.path.insert(0, sys.argv[1])
import numpy as np, torch
import boosters_b200 as bst
from boosters_b200 import _native
tree = {"group": 0, "split_index": np.array([1, 0, 0]), "threshold": np.zeros(3, np.float32),
        "left": np.array([1, 0, 0]), "right": np.array([2, 0, 0]), "default_left": np.zeros(3, int),
        "is_leaf": np.array([0, 1, 1], np.uint8), "leaf_value": np.array([0, 1, 2], np.float32)}
few, many = (bst.GBDTModel.from_trees(3, [tree] * t, bst.Objective.squared(), (0.0,)) for t in (96, 600))

def run(m, x, out):
    _native.check(_native.lib.bst_gbdt_predict_device(
        m._h, ctypes.c_void_p(x.data_ptr()), x.shape[0], 3, 1, ctypes.c_void_p(out.data_ptr()),
        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    torch.cuda.synchronize()

x = torch.randn((18_000, 3), device="cuda")  # 18,048 x 600 leaf values: 43 MB; bins: 0.1 MB
out = torch.empty((1, 18_000), device="cuda")
want = torch.where(x[:, 1] < 0, 600.0, 1200.0)
run(many, x[:100].contiguous(), out[:, :100].contiguous())  # the forests, the kernels, the pool's first block
run(few, torch.zeros((200_000, 3), device="cuda"), torch.empty((1, 200_000), device="cuda"))
hold, size = [], 1 << 34
while size >= 1 << 21:  # all of the device but a few MB
    try:
        hold.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
    except torch.OutOfMemoryError:
        size >>= 1
free = torch.cuda.mem_get_info()[0] >> 20
try:
    run(many, x, out)
    print("free", free, "equal", bool((out[0] == want).all()))
except _native.BoostersError as e:
    print("free", free, "error", e)
"""


def test_prediction_without_room_for_leaf_values():
    r = subprocess.run([sys.executable, "-c", PREDICT, ROOT], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    line = next(ln for ln in r.stdout.split("\n") if ln.startswith("free"))
    assert int(line.split()[1]) < 40, line  # less than the leaf values take
    assert line.endswith("equal True"), line
