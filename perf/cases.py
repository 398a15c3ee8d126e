"""Workloads of the engine's speed measurements: training, prediction and serving.

Each case is one call a program makes through the public interface, over the
sizes the benchmark, the tests and the reference's published tables use:
training runs from a few thousand to a million rows (depth-wise and leaf-wise,
every gradient precision, categorical columns, sampling and early stopping),
batch prediction of host and device rows, and served requests from one small
batch to a burst of mixed sizes.
"""
import ctypes

import numpy as np
import torch

import boosters_b200 as bst
from boosters_b200 import _native

DEVICE = "cuda:0"


# ---- cases -------------------------------------------------------------------

def listed():
    return [
        # the reference's smallest training table row: latency of short trees
        _train("train_reg_5k", "squared", 5_000, 100, trees=50, depth=6),
        # its 50k x 100 row with every default (f32 histograms)
        _train("train_reg_50k", "squared", 50_000, 100, trees=50, depth=6),
        # the benchmark's workload in its fastest form, one whole model
        _train("train_bin_1m_q8", "logistic", 1_000_000, 100, trees=100, depth=8, nan_cols=20, precision="q8",
               pinned=True),
        # the same data with the default precision
        _train("train_bin_1m_fp32", "logistic", 1_000_000, 100, trees=50, depth=8, nan_cols=20, pinned=True),
        # best-first growth to 255 leaves on wide data
        _train("train_leafwise_1m", "logistic", 1_000_000, 200, trees=12, leaves=255, nan_cols=20, precision="q16",
               pinned=True),
        # multiclass with categorical columns: ten trees a round
        _train("train_multi_200k", "softmax", 200_000, 40, cats=10, classes=10, trees=10, depth=6),
        # a tuned run: row and column sampling, validation rows, early stopping
        _train("train_tuned_100k", "logistic", 100_000, 51, trees=60, depth=6, subsample=0.8, colsample=0.8,
               val_rows=25_000, stopping=15),
        # scoring a small batch of host rows, the reference's table row
        _predict("predict_host_1k", 1_000, 100, trees=200, depth=6),
        # scoring a whole table of host rows
        _predict("predict_host_300k", 300_000, 100, trees=500, depth=8),
        # device-resident rows: a feature pipeline that ends on the GPU
        _predict("predict_device_100k", 100_003, 100, trees=1000, depth=8, where="device"),
        # one small request to a server: latency
        _serve("serve_one", 1, 16, 100, trees=1000, depth=8, where="host"),
        # a burst of requests of mixed sizes, device rows: throughput
        _serve("serve_burst", 48, 65_536, 100, trees=1000, depth=8, where="device"),
    ]


def _train(name, objective, rows, numeric, *, cats=0, classes=1, trees, depth=0, leaves=0, nan_cols=0,
           precision="fp32", subsample=1.0, colsample=1.0, val_rows=0, stopping=0, pinned=False):
    return {"name": name, "kind": "train", "objective": objective, "rows": rows, "numeric": numeric, "cats": cats,
            "classes": classes, "trees": trees, "depth": depth, "leaves": leaves, "nan_cols": nan_cols,
            "precision": precision, "subsample": subsample, "colsample": colsample, "val_rows": val_rows,
            "stopping": stopping, "pinned": pinned}


def _predict(name, rows, features, *, trees, depth, where="host"):
    return {"name": name, "kind": "predict", "rows": rows, "features": features, "trees": trees, "depth": depth,
            "where": where}


def _serve(name, requests, max_rows, features, *, trees, depth, where):
    return {"name": name, "kind": "serve", "requests": requests, "max_rows": max_rows, "features": features,
            "trees": trees, "depth": depth, "where": where}


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["train_depthwise", "train_leafwise", "train_multi", "train_tuned", "predict", "predict",
                       "serve"])
    if kind == "train_depthwise":
        c = _train("", rng.choice(["squared", "logistic"]), _log_int(rng, 2_000, 700_000), rng.randint(13, 128),
                   trees=rng.randint(20, 60), depth=rng.randint(4, 8), nan_cols=rng.choice([0, 5, 13]),
                   precision=rng.choice(["fp32", "fp32", "q8", "q16"]), pinned=rng.random() < 0.5)
    elif kind == "train_leafwise":
        c = _train("", rng.choice(["squared", "logistic"]), _log_int(rng, 5_000, 500_000), rng.randint(20, 160),
                   trees=rng.randint(6, 12), leaves=rng.choice([31, 63, 100, 255]), nan_cols=rng.choice([0, 7]),
                   precision=rng.choice(["fp32", "q16", "q8"]))
    elif kind == "train_multi":
        c = _train("", "softmax", _log_int(rng, 3_000, 150_000), rng.randint(10, 50), cats=rng.randint(1, 12),
                   classes=rng.randint(3, 10), trees=rng.randint(4, 10), depth=rng.randint(4, 7),
                   precision=rng.choice(["fp32", "fp32", "q8"]))
    elif kind == "train_tuned":
        rows = _log_int(rng, 5_000, 80_000)
        c = _train("", rng.choice(["squared", "logistic"]), rows, rng.randint(13, 90), trees=rng.randint(25, 60),
                   depth=rng.randint(4, 7), subsample=rng.choice([0.6, 0.8, 1.0]),
                   colsample=rng.choice([0.7, 0.8, 1.0]), val_rows=rows // 4, stopping=rng.randint(8, 20))
    elif kind == "predict":
        c = _predict("", _log_int(rng, 1, 250_000), rng.randint(13, 128), trees=rng.randint(50, 600),
                     depth=rng.randint(4, 8), where=rng.choice(["host", "device"]))
    else:
        c = _serve("", _log_int(rng, 1, 40), _log_int(rng, 8, 50_000), rng.randint(13, 120),
                   trees=rng.randint(100, 900), depth=rng.randint(5, 8), where=rng.choice(["host", "device"]))
    del c["name"]
    return c


# ---- inputs ------------------------------------------------------------------

def _generator(seed):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(int(seed))
    return g


def _table(case, seed, rows):
    """Feature-major f32 columns and targets, on the GPU."""
    g = _generator(seed)
    n_num, n_cat = case["numeric"], case["cats"]
    x = torch.empty((n_num + n_cat, rows), dtype=torch.float32, device=DEVICE)
    half = n_num // 2
    x[:half].normal_(generator=g)
    if case["objective"] == "logistic":  # half normal, half uniform
        x[half:n_num].uniform_(generator=g)
    else:
        x[half:n_num].normal_(generator=g)
    for c in range(n_num, n_num + n_cat):  # Zipf-distributed categories
        card = int(torch.randint(4, 65, (1,), generator=g, device=DEVICE))
        p = 1.0 / torch.arange(1, card + 1, device=DEVICE, dtype=torch.float64) ** 1.2
        cdf = torch.cumsum(p / p.sum(), 0)
        u = torch.rand(rows, generator=g, device=DEVICE, dtype=torch.float64)
        x[c] = torch.searchsorted(cdf, u).clamp_(max=card - 1).float()
    if case["objective"] == "squared":
        k = min(20, n_num)
        w = torch.randn(k, generator=g, device=DEVICE)
        y = w @ x[:k] + 0.1 * torch.randn(rows, generator=g, device=DEVICE)
    elif case["objective"] == "logistic":
        m = 0.5 * torch.randn(rows, generator=g, device=DEVICE)
        for i in range(min(10, n_num // 2)):
            m += x[i] * x[n_num - 1 - i]
        y = (torch.rand(rows, generator=g, device=DEVICE) < torch.sigmoid(m)).float()
    else:
        w = torch.randn((case["classes"], n_num + n_cat), generator=g, device=DEVICE) / 4.0
        w[:, n_num:] /= 8.0
        u = torch.rand((case["classes"], rows), generator=g, device=DEVICE).clamp_(1e-6, 1.0 - 1e-6)
        y = torch.argmax(w @ x - torch.log(-torch.log(u)), 0).float()
    for c in range(min(case["nan_cols"], n_num)):  # a tenth of these columns is missing
        x[c].masked_fill_(torch.rand(rows, generator=g, device=DEVICE) < 0.1, float("nan"))
    return x, y


def _host(t, pinned):
    if not pinned:
        return t.cpu().numpy()
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    return h.numpy()


def _trees(case, seed):
    """Random trees as training leaves them: thresholds on a grid of 255
    quantile bounds a feature, some branches ending early."""
    rng = np.random.default_rng(int(seed))
    depth, n_trees, F = case["depth"], case["trees"], case["features"]
    n = 2 ** (depth + 1) - 1
    level = np.floor(np.log2(np.arange(1, n + 1))).astype(np.int64)
    grid = np.sort(rng.standard_normal((F, 255)).astype(np.float32), axis=1)
    trees = []
    for _ in range(n_trees):
        leaf = (level == depth) | ((level >= 3) & (rng.random(n) < 0.06))
        alive = np.ones(n, bool)
        for lv in range(1, depth + 1):  # no node below a leaf
            i = np.arange(2 ** lv - 1, 2 ** (lv + 1) - 1)
            p = (i - 1) // 2
            alive[i] = alive[p] & ~leaf[p]
        new = np.cumsum(alive) - 1
        keep = np.flatnonzero(alive)
        lf = leaf[keep]
        feat = rng.integers(0, F, keep.size)
        child = np.minimum(2 * keep + 1, n - 2)
        trees.append({
            "split_index": np.where(lf, 0, feat).astype(np.uint32),
            "threshold": np.where(lf, 0, grid[feat, rng.integers(0, 255, keep.size)]).astype(np.float32),
            "left": np.where(lf, 0, new[child]).astype(np.uint32),
            "right": np.where(lf, 0, new[child + 1]).astype(np.uint32),
            "default_left": rng.integers(0, 2, keep.size).astype(np.uint8),
            "is_leaf": lf.astype(np.uint8),
            "leaf_value": np.where(lf, 0.05 * rng.standard_normal(keep.size), 0).astype(np.float32),
        })
    return trees


def _rows(case, seed, rows):
    """Sample-major f32 rows on the GPU, a tenth of a fifth of the columns missing."""
    g = _generator(seed)
    x = torch.randn((rows, case["features"]), generator=g, device=DEVICE)
    k = case["features"] // 5
    miss = torch.rand((rows, k), generator=g, device=DEVICE) < 0.1
    x[:, :k].masked_fill_(miss, float("nan"))
    return x


def _request_sizes(case):
    """Row counts spread over the logarithm of 1 .. max_rows, in a fixed mixed order."""
    if case["requests"] == 1:
        return [case["max_rows"]]
    q = (np.arange(case["requests"]) + 0.5) / case["requests"]
    sizes = np.maximum(1, np.round(case["max_rows"] ** q)).astype(np.int64)
    return [int(v) for v in np.random.default_rng(7).permutation(sizes)]


def _config(case):
    objective = {"squared": bst.Objective.squared, "logistic": bst.Objective.logistic,
                 "softmax": lambda: bst.Objective.softmax(case["classes"])}[case["objective"]]()
    kw = {}
    if case["leaves"]:
        kw.update(growth_strategy=bst.GrowthStrategy.Leafwise, n_leaves=case["leaves"])
    else:
        kw.update(max_depth=case["depth"])
    if case["stopping"]:
        kw.update(early_stopping_rounds=case["stopping"])
    return bst.GBDTConfig(n_estimators=case["trees"], learning_rate=0.1, objective=objective,
                          precision=case["precision"], subsample=case["subsample"],
                          colsample_bytree=case["colsample"], **kw)


def prepare(case, seed):
    if case["kind"] == "train":
        cats = list(range(case["numeric"], case["numeric"] + case["cats"]))
        total = case["rows"] + case["val_rows"]
        x, y = _table(case, seed, total)
        n = case["rows"]
        ds = bst.Dataset.from_feature_major(_host(x[:, :n].contiguous(), case["pinned"]),
                                            _host(y[:n].contiguous(), case["pinned"]), categorical_features=cats)
        val = None
        if case["val_rows"]:
            val = bst.Dataset.from_feature_major(_host(x[:, n:].contiguous(), False), _host(y[n:], False),
                                                 categorical_features=cats)
        nodes = 2 * case["leaves"] - 1 if case["leaves"] else 2 ** (case["depth"] + 1) - 1
        return {"kind": "train", "ds": ds, "val": val, "config": _config(case),
                "size": (case["trees"] * case["classes"], nodes)}
    model = bst.GBDTModel.from_trees(case["features"], _trees(case, seed), bst.Objective.logistic(), (0.1,))
    if case["kind"] == "predict":
        x = _rows(case, seed, case["rows"])
        if case["where"] == "host":
            return {"kind": "predict", "model": model, "ds": bst.Dataset(x.cpu().numpy())}
        return {"kind": "predict_device", "model": model, "x": x,
                "out": torch.empty((1, case["rows"]), dtype=torch.float32, device=DEVICE)}
    reqs, outs = [], []
    for i, n in enumerate(_request_sizes(case)):
        x = _rows(case, seed * 1000 + i, n)
        if case["where"] == "host":
            reqs.append(x.cpu().numpy())
            outs.append(np.empty((1, n), np.float32))
        else:
            reqs.append(x)
            outs.append(torch.empty((1, n), dtype=torch.float32, device=DEVICE))
    torch.cuda.synchronize()
    return {"kind": "serve", "server": bst.PredictionServer(model), "requests": reqs, "outs": outs}


# ---- one pass ----------------------------------------------------------------

def _tree_arrays(model, n_trees, max_nodes):
    """Every tree's nodes as one [n_trees, max_nodes] array a field, zeros
    where a tree has fewer nodes or training stopped early."""
    lib, fields = _native.lib, {}
    for k, d in _FIELDS:
        fields[k] = np.zeros((n_trees, max_nodes), d)
    for t in range(model.n_trees):
        ptrs = [ctypes.cast(a.ctypes.data + t * a.strides[0], _POINTERS[a.dtype]) for a in fields.values()]
        _native.check(lib.bst_model_tree_nodes(model._h, t, *ptrs))
    return dict(fields, kept=model.n_trees)


_FIELDS = [("split_index", np.uint32), ("threshold", np.float32), ("left", np.uint32), ("right", np.uint32),
           ("default_left", np.uint8), ("is_leaf", np.uint8), ("leaf_value", np.float32), ("split_type", np.uint8),
           ("gain", np.float32), ("cover", np.float32)]
_POINTERS = {np.dtype(np.uint32): ctypes.POINTER(ctypes.c_uint32), np.dtype(np.float32): ctypes.POINTER(ctypes.c_float),
             np.dtype(np.uint8): ctypes.POINTER(ctypes.c_uint8)}


def run(state):
    kind = state["kind"]
    if kind == "train":
        model = bst.GBDTModel.train(state["ds"], state["config"], val_set=state["val"])
        return dict(_tree_arrays(model, *state["size"]), predictions=model.train_predictions())
    if kind == "predict":
        return state["model"].predict(state["ds"])
    if kind == "predict_device":
        x, out = state["x"], state["out"]
        _native.check(_native.lib.bst_gbdt_predict_device(
            state["model"]._h, ctypes.c_void_p(x.data_ptr()), x.shape[0], x.shape[1], 0,
            ctypes.c_void_p(out.data_ptr()), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
        return out
    server = state["server"]
    tickets = [server.submit(r, o) for r, o in zip(state["requests"], state["outs"])]
    return [server.wait(t) for t in tickets]


def work(case):
    """Bytes: the raw table read once; per tree, one read of the rows' bins
    (a byte each) and gradients and one update of the predictions; for
    prediction the rows, the trees and the results. Flops: a tree's gradient
    and hessian additions over one level, or a comparison per tree level."""
    if case["kind"] == "train":
        F, n, G = case["numeric"] + case["cats"], case["rows"], case["classes"]
        trees = case["trees"] * G
        return {"bytes": 4 * (n + case["val_rows"]) * (F + 1) + trees * n * (F + 16) + 4 * n * G,
                "flops": 2 * trees * n * F}
    rows = case["rows"] if case["kind"] == "predict" else sum(_request_sizes(case))
    nodes = case["trees"] * (2 ** case["depth"])
    return {"bytes": 4 * rows * (case["features"] + 1) + 8 * nodes, "flops": rows * case["trees"] * (case["depth"] + 1)}


# ---- 64-bit values -------------------------------------------------------------

def _exact_rows(trees, x):
    """sigmoid(0.1 + the trees' leaves), summed in f64, for sample-major f32 rows."""
    total = torch.full((x.shape[0],), float(np.float32(0.1)), dtype=torch.float64, device=x.device)
    for t in trees:
        a = {k: torch.from_numpy(v.astype(np.int64) if v.dtype.kind == "u" else v).to(x.device)
             for k, v in t.items()}
        node = torch.zeros(x.shape[0], dtype=torch.int64, device=x.device)
        for _ in range(32):
            if bool(a["is_leaf"][node].all()):
                break
            v = x.gather(1, a["split_index"][node][:, None])[:, 0]
            go_left = torch.where(torch.isnan(v), a["default_left"][node] != 0, v < a["threshold"][node])
            child = torch.where(go_left, a["left"][node], a["right"][node])
            node = torch.where(a["is_leaf"][node] != 0, node, child)
        total += a["leaf_value"][node].double()
    return torch.sigmoid(total)


def exact(case, seed):
    if case["kind"] == "train":  # a whole model: no closed form
        return None
    trees = _trees(case, seed)
    if case["kind"] == "predict":
        p = _exact_rows(trees, _rows(case, seed, case["rows"]))
        return p.cpu().numpy()[:, None] if case["where"] == "host" else p[None, :]
    sizes = _request_sizes(case)
    xs = [_rows(case, seed * 1000 + i, n) for i, n in enumerate(sizes)]
    p = _exact_rows(trees, torch.cat(xs))
    return [q[None, :].cpu().numpy() if case["where"] == "host" else q[None, :] for q in torch.split(p, sizes)]
