"""The bounds-checked library over the level kernels: training sets past the one
launch a tree, in FP32, with categorical columns and several outputs, and with
columns of more than 264 bins (the general tiles); no check fails, and trees and
predictions equal the normal library's."""
import json
import os
import subprocess
import sys

import numpy as np
import pytest

import boosters_b200 as bst
from test_gpu_checked import CHECKED, ROOT

pytestmark = pytest.mark.gpu

CASES = {
    "fp32": dict(precision="fp32", max_depth=8),
    "q16_columns_of_few_and_many_bins": dict(precision="q16", max_depth=6, max_bins=600),
    "softmax_categories": dict(precision="q8", max_depth=6, softmax=4),
    "fp32_categories_sampling": dict(precision="fp32", max_depth=5, softmax=3, subsample=0.7, colsample_bytree=0.8),
}

CHILD = r"""
import ctypes, json, sys
import numpy as np
sys.path[:0] = [sys.argv[1], sys.argv[1] + "/tests"]
import test_gpu_checked_levels as t
from boosters_b200 import _native as n
assert n.LIB_PATH.endswith("libboosters_b200_checked.so"), n.LIB_PATH
report = {}
for name in t.CASES:
    np.savez(f"{sys.argv[2]}/{name}.npz", **t.run_case(name))
    v, site, idx, bound = ctypes.c_uint64(), ctypes.c_uint32(), ctypes.c_uint64(), ctypes.c_uint64()
    rc = n.lib.bst_check_report(0, ctypes.byref(v), ctypes.byref(site), ctypes.byref(idx), ctypes.byref(bound))
    report[name] = dict(rc=rc, violations=v.value, site=site.value, index=idx.value, bound=bound.value)
json.dump(report, open(f"{sys.argv[2]}/report.json", "w"))
"""


def run_case(name):
    c = dict(CASES[name])
    n = 130_000
    if "softmax" in c:
        x, y = bst.synth.multiclass(n, n_numeric=12, n_categorical=4, n_classes=c["softmax"], seed=5)
        cats, objective = list(range(12, 16)), bst.Objective.softmax(c.pop("softmax"))
    else:
        x, y = bst.synth.binary(n, 24, n_nan_cols=4, seed=13)
        x[5] = np.round(2 * x[5])
        cats, objective = [], bst.Objective.logistic()
    ds = bst.Dataset.from_feature_major(x, y, categorical_features=cats)
    m = bst.GBDTModel.train(ds, bst.GBDTConfig(objective=objective, n_estimators=3, learning_rate=0.3, **c),
                            n_threads=1, record_leaves=True)
    assert not m.tune_info.startswith("one launch"), m.tune_info
    keys = ("split_index", "split_bin", "left", "right", "default_left", "is_leaf", "split_type", "cat_words",
            "leaf_value")
    out = {k: np.concatenate([np.asarray(m.tree(i)[k]).ravel() for i in range(m.n_trees)]) for k in keys}
    out["rows"] = np.concatenate([np.asarray(m.tree_row_leaves(i, n)).ravel() for i in range(m.n_trees)])
    out["pred"] = np.asarray(m.predict_group_major(ds)).ravel()
    return out


@pytest.fixture(scope="module")
def checked_dir(tmp_path_factory):
    if not os.path.exists(CHECKED):
        pytest.fail("libboosters_b200_checked.so is not built (python -m boosters_b200.build --checked)")
    out = tmp_path_factory.mktemp("checked_levels")
    r = subprocess.run([sys.executable, "-c", CHILD, ROOT, str(out)], env=dict(os.environ, BST_LIBRARY="checked"),
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]
    return out


@pytest.mark.parametrize("name", list(CASES))
def test_checked_levels_match_and_record_nothing(checked_dir, name):
    got = json.load(open(checked_dir / "report.json"))[name]
    assert got["rc"] == 0 and got["violations"] == 0, got
    chk = np.load(checked_dir / f"{name}.npz")
    for k, v in run_case(name).items():
        np.testing.assert_array_equal(chk[k], v, err_msg=f"{name}: {k}")
