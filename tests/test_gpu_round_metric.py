"""Every metric of an early-stopped run, evaluated on the device each round,
stops and truncates where the same rule on the host's metric of prefix models
does, with weights, several outputs, categorical splits and row counts at the
edges of the evaluation's blocks."""
import numpy as np
import pytest

import boosters_b200 as bst
from test_gpu_early_stopping import prefix_model

pytestmark = pytest.mark.gpu

O, M = bst.Objective, bst.Metric
CASES = {
    "rmse": (O.squared(), M.rmse(), {}), "mae": (O.squared(), M.mae(), {}), "mape": (O.squared(), M.mape(), {}),
    "huber": (O.squared(), M.huber(0.7), {"delta": 0.7}),
    "quantile": (O.pinball([0.2, 0.5, 0.9]), M.quantile([0.2, 0.5, 0.9]), {"alpha": [0.2, 0.5, 0.9]}),
    "poisson": (O.poisson(), M.poisson_deviance(), {}), "logloss": (O.logistic(), M.logloss(), {}),
    "margin_accuracy": (O.hinge(), M.margin_accuracy(), {}), "mlogloss": (O.softmax(4), M.mlogloss(), {}),
}


def rule(values, patience, higher):
    best, best_round, cur, best_n, run = None, 0, 0, 0, 0
    for r, v in enumerate(values):
        run = r + 1
        improved = best is None or (v > best if higher else v < best)
        if improved:
            best, best_round = v, cur
        cur += 1
        if cur - best_round > patience:
            break
        if improved:
            best_n = r + 1
    return best_n if 0 < best_n < run else run


@pytest.mark.parametrize("kind", list(CASES))
@pytest.mark.parametrize("nv", [1, 255, 257, 1500])
def test_stops_where_the_host_metric_does(kind, nv):
    objective, metric, extra = CASES[kind]
    rng = np.random.default_rng(nv)
    n, cats = 1200, [5]
    x = rng.standard_normal((6, n + nv)).astype(np.float32)
    x[5] = rng.integers(0, 9, n + nv)
    x[1][rng.random(n + nv) < 0.1] = np.nan
    z = x[0] + (x[5] > 4) + 0.8 * rng.standard_normal(n + nv)
    y = {"poisson": lambda: rng.poisson(np.exp(np.clip(z, -2, 2))), "logloss": lambda: z > 0.3,
         "margin_accuracy": lambda: z > 0.3, "mlogloss": lambda: np.clip(z + 1, 0, 3).astype(int)}.get(kind, lambda: z)()
    y = np.asarray(y, np.float32)
    w = rng.uniform(0.2, 3.0, n + nv).astype(np.float32)
    ds = bst.Dataset.from_feature_major(x[:, :n].copy(), y[:n], weights=w[:n], categorical_features=cats)
    dv = bst.Dataset.from_feature_major(x[:, n:].copy(), y[n:], weights=w[n:], categorical_features=cats)
    kw = dict(objective=objective, metric=metric, n_estimators=25, max_depth=5, learning_rate=0.6)
    full = bst.GBDTModel.train(ds, bst.GBDTConfig(**kw))
    groups, raw = objective.n_outputs, kind == "margin_accuracy"
    values = [bst.metric(kind, prefix_model(full, r, groups).predict_group_major(dv, raw=raw), y[n:], w[n:], **extra)
              for r in range(1, 26)]
    es = bst.GBDTModel.train(ds, bst.GBDTConfig(early_stopping_rounds=3, **kw), val_set=dv)
    assert es.n_trees == groups * rule(values, 3, raw), values
