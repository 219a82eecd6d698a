"""What this framework is used for, as cases that can be timed and compared: training a model on a table and applying it.

A case is a plain dict; ``kind`` names the path:

* ``fit``   -- ``CatBoost.fit`` on a ``Pool`` in host memory, then the trained model's raw predictions for rows it has not
               seen.  Everything a fit does is inside a pass: upload, binning, all boosting iterations, the finished model.
               Options: loss (binary, regression, five classes, ranking), weights, an evaluation set, categorical columns,
               mostly-zero columns, depth-wise growth, 16 to 254 borders.
* ``serve`` -- ``predict(task_type='GPU')`` of a stored model on rows in host memory: from a handful of rows per call (an
               online service) to batches where the transfer counts.
* ``score`` -- ``GpuPredictor.predict_device``: the rows are already on the GPU.

``prepare`` makes host tables (that is what ``fit`` and ``predict`` take); they are drawn on the GPU and copied over.
"""
from __future__ import annotations

import json
import math

import numpy as np
import torch

import catboost_b200 as cb
from catboost_b200.models.gpu_apply import GpuPredictor

_FIT = dict(kind="fit", rows=0, cols=0, trees=0, depth=6, borders=128, loss="Logloss", zeros=0.0, cats=0, weighted=False,
            eval_rows=0, policy="SymmetricTree", bootstrap="Bayesian", ready=True, pinned=False)
_APPLY = dict(kind="serve", rows=0, cols=0, trees=0, depth=6, borders=128, dims=1)


def listed():
    return [
        # somebody trying things out: a few thousand rows, arrays handed straight to fit(); launches and host work count
        dict(_FIT, name="fit small arrays", rows=3_000, cols=12, trees=100, ready=False),
        # the everyday regression run: odd sizes, document weights, the finest border grid, an evaluation set that is
        # scored after every tree
        dict(_FIT, name="fit regression eval", rows=60_013, cols=39, trees=100, depth=8, borders=254, loss="RMSE",
             weighted=True, eval_rows=10_007, bootstrap="Bernoulli"),
        # a mid-sized table, the shape of the web-search set in the reference's training-speed table
        dict(_FIT, name="fit 1.2M x 137", rows=1_200_000, cols=137, trees=100, pinned=True),
        # the headline benchmark's table
        dict(_FIT, name="fit 10.5M x 28", rows=10_500_000, cols=28, trees=150, pinned=True),
        # many columns, few rows
        dict(_FIT, name="fit 100K x 2000", rows=100_003, cols=2_000, trees=100, pinned=True),
        # learning to rank on mostly-zero columns: query-wise derivatives, 64 borders
        dict(_FIT, name="fit ranking sparse", rows=200_000, cols=300, trees=20, borders=64, loss="YetiRank", zeros=0.6),
        # five classes
        dict(_FIT, name="fit 5 classes", rows=300_000, cols=60, trees=100, loss="MultiClass"),
        # numeric and categorical columns: target statistics, many columns of 16 bins, deep trees
        dict(_FIT, name="fit categorical", rows=400_000, cols=13, cats=8, trees=80, depth=8),
        # an online service: one small batch per call
        dict(_APPLY, name="serve 200 rows", rows=200, cols=28, trees=500),
        # batch apply from ordinary (pageable) host memory
        dict(_APPLY, name="serve 1M rows", rows=1_000_003, cols=28, trees=500),
        # rows already on the GPU, a full-sized model
        dict(_APPLY, kind="score", name="score 4M x 28", rows=4_000_000, cols=28, trees=1_000),
        # rows already on the GPU, many columns, a model that uses most of them
        dict(_APPLY, kind="score", name="score 1M x 700", rows=1_000_000, cols=700, trees=200, borders=64),
    ]


def _between(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fit", "fit", "fit", "fit", "serve", "score"])
    if kind == "fit":
        loss = rng.choice(["Logloss", "Logloss", "RMSE", "MultiClass", "YetiRank"])
        rows = _between(rng, 2_000, 4_000_000)
        cols = _between(rng, 5, max(6, min(2_000, 160_000_000 // rows)))
        c = dict(_FIT, rows=rows, cols=cols, loss=loss, depth=rng.choice([4, 6, 6, 7, 8]),
                 borders=rng.choice([32, 64, 128, 128, 254]), bootstrap=rng.choice(["Bayesian", "Bernoulli", "No"]),
                 zeros=rng.choice([0.0, 0.0, 0.6]), weighted=rng.random() < 0.3 and loss != "YetiRank",
                 eval_rows=rng.choice([0, 0, 5_003]) if loss != "YetiRank" else 0, ready=rng.random() < 0.7)
        if loss == "Logloss" and rows <= 400_000 and rng.random() < 0.3:
            c["cats"] = rng.randint(1, 8)
            c["cols"] = min(c["cols"], 40)
        # as many trees as keep a pass well below the largest listed one
        c["trees"] = max(10, min(100, int(6e9 / (rows * (c["cols"] + 20 * c["cats"] + 20) * (3 if loss == "MultiClass" else 1)))))
        if loss == "YetiRank":
            c["trees"] = min(c["trees"], 20)
        return c
    cols = _between(rng, 5, 800)
    rows = _between(rng, 1, 2_000_000) if kind == "serve" else _between(rng, 1_000, 4_000_000)
    return dict(_APPLY, kind=kind, rows=max(1, min(rows, 250_000_000 // cols)), cols=cols, trees=_between(rng, 50, 1_000),
                depth=rng.choice([4, 6, 6, 8]), borders=rng.choice([32, 64, 128, 254]), dims=rng.choice([1, 1, 3]))


# ---------------------------------------------------------------------------------------------------------
def _host(t, pinned=False):
    if not pinned:
        return t.cpu().numpy()
    out = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    out.copy_(t)
    return out.numpy()


def _table(case, rows, gen, pinned=False):
    """Columns of different kinds -- normal, skewed counts, uniform -- and a target that depends on some of them."""
    dev = torch.device("cuda")
    F = case["cols"]
    X = torch.randn((rows, F), generator=gen, device=dev)
    X[:, 1::5] = X[:, 1::5].abs()
    if F > 3:
        X[:, 3::7] = torch.floor(torch.exp(X[:, 3::7] + 1.0))
    if case.get("zeros"):
        X = torch.where(torch.rand((rows, F), generator=gen, device=dev) < case["zeros"], torch.zeros((), device=dev), X.abs())
    wgen = torch.Generator(device=dev).manual_seed(77)           # the law of the data, the same for every table
    k = min(F, 24)
    w = torch.randn(k, generator=wgen, device=dev) * (0.85 ** torch.arange(k, device=dev))
    Z = torch.tanh(X[:, :k])
    f = Z @ w
    f += 0.8 * Z[:, 0] * Z[:, 1 % F] - 0.6 * Z[:, 2 % F].abs() * Z[:, 0]
    return X, f / f.std().clamp_min(1e-6)


def _target(case, f, gen):
    dev = f.device
    if case["loss"] == "RMSE":
        return 3.0 * f + torch.randn(f.shape, generator=gen, device=dev)
    if case["loss"] in ("MultiClass", "YetiRank"):
        s = f + 0.4 * torch.randn(f.shape, generator=gen, device=dev)
        q = [-0.9, -0.2, 0.3, 1.0] if case["loss"] == "MultiClass" else [0.0, 0.8, 1.4, 2.0]
        return torch.bucketize(s, torch.tensor(q, device=dev)).float()
    return (torch.rand(f.shape, generator=gen, device=dev) < torch.sigmoid(2.0 * f)).float()


def _frame(case, X, f, gen):
    """The table with categorical columns behind the numeric ones (integer codes, skewed frequencies, each with an effect)."""
    import pandas as pd
    dev = f.device
    cols = {f"n{j}": _host(X[:, j].contiguous()) for j in range(X.shape[1])}
    wgen = torch.Generator(device=dev).manual_seed(78)
    for j in range(case["cats"]):
        card = int(10 * 8 ** (j / 2.0))
        code = torch.floor(card * torch.rand(f.shape, generator=gen, device=dev) ** 3.0).clamp_(max=card - 1).long()
        f = f + 0.5 * torch.randn(card, generator=wgen, device=dev)[code]
        cols[f"c{j}"] = _host(code.int())
    return pd.DataFrame(cols), f, [f"c{j}" for j in range(case["cats"])]


def _prepare_fit(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    held = min(20_000, max(500, case["rows"] // 4)) if not case["cats"] else 2_000
    pools = []
    for part, rows in (("train", case["rows"]), ("eval", case["eval_rows"]), ("held", held)):
        if rows == 0:
            pools.append(None)
            continue
        X, f = _table(case, rows, gen)
        cats = None
        if case["cats"]:
            data, f, cats = _frame(case, X, f, gen)
        else:
            data = _host(X, case["pinned"] and part == "train")
        y = _host(_target(case, f, gen))
        weight = _host(torch.rand(rows, generator=gen, device="cuda") + 0.5) if case["weighted"] else None
        group = None
        if case["loss"] == "YetiRank":
            sizes = np.random.default_rng(int(seed)).integers(5, 201, size=rows // 5 + 1)
            group = np.repeat(np.arange(len(sizes)), sizes)[:rows]
        if part == "held":
            pools.append(cb.Pool(data, cat_features=cats))
        elif part == "train" and not case["ready"]:
            pools.append(dict(X=data, y=y, cat_features=cats, sample_weight=weight, group_id=group))
        else:
            pools.append(cb.Pool(data, y, weight=weight, group_id=group, cat_features=cats))
            if part == "train":
                pools[-1].quantize(border_count=case["borders"])
    torch.cuda.empty_cache()
    params = dict(loss_function=case["loss"], iterations=case["trees"], depth=case["depth"], border_count=case["borders"],
                  learning_rate=0.1, task_type="GPU", devices="0", random_seed=int(seed) % 1000, bootstrap_type=case["bootstrap"],
                  grow_policy=case["policy"], use_best_model=False, allow_writing_files=False, verbose=False)
    if case["cats"]:
        params["max_ctr_complexity"] = 2
    return dict(case=case, train=pools[0], eval=pools[1], held=pools[2], params=params)


def _trees(case, seed):
    """Random splits over a grid of borders, leaf values that shrink: (grid, split features, split borders, leaf values)."""
    rng = np.random.default_rng(int(seed))
    F, T, D, dims = case["cols"], case["trees"], case["depth"], case["dims"]
    grid = np.sort(rng.standard_normal((F, case["borders"])).astype(np.float32), axis=1)
    feat = rng.integers(0, F, (T, D))
    pick = rng.integers(0, case["borders"], (T, D))
    vals = rng.standard_normal((T, (1 << D) * dims)) * 0.1 / (1.0 + np.arange(T)[:, None] / 100.0)
    return grid, feat, pick, vals


def _stored_model(case, seed):
    """A model as a service loads it from a file."""
    F, T, D, dims = case["cols"], case["trees"], case["depth"], case["dims"]
    grid, feat, pick, vals = _trees(case, seed)
    doc = {"features_info": {"float_features": [
        {"feature_index": j, "flat_feature_index": j, "borders": grid[j].tolist(), "has_nans": False,
         "nan_value_treatment": "AsIs", "feature_id": str(j)} for j in range(F)]},
        "scale_and_bias": [1.0, [0.1] * dims],
        "model_info": {"loss_name": "RMSE" if dims == 1 else "MultiRMSE", "class_names": None, "dims": dims, "n_features": F,
                       "feature_names": [str(j) for j in range(F)], "params": {}},
        "oblivious_trees": [{"splits": [{"split_type": "FloatFeature", "float_feature_index": int(feat[t, d]),
                                         "border": float(grid[feat[t, d], pick[t, d]])} for d in range(D)],
                             "leaf_values": vals[t].tolist(), "leaf_weights": [1.0] * (1 << D)} for t in range(T)]}
    return cb.CatBoost().load_model(blob=json.dumps(doc).encode(), format="json")


def _rows(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    return torch.randn((case["rows"], case["cols"]), generator=gen, device="cuda")


def prepare(case, seed):
    if case["kind"] == "fit":
        return _prepare_fit(case, seed)
    model = _stored_model(case, seed)
    X = _rows(case, seed)
    if case["kind"] == "score":
        return dict(case=case, model=model, predictor=GpuPredictor(model._model), X=X)
    return dict(case=case, model=model, X=_host(X))


def run(state):
    case = state["case"]
    if case["kind"] == "score":
        return state["predictor"].predict_device(state["X"])
    if case["kind"] == "serve":
        return state["model"].predict(state["X"], prediction_type="RawFormulaVal", task_type="GPU")
    model = cb.CatBoost(state["params"])
    if isinstance(state["train"], dict):
        model.fit(**state["train"], eval_set=state["eval"])
    else:
        model.fit(state["train"], eval_set=state["eval"])
    curves = model.get_evals_result()
    return {"raw": model.predict(state["held"], prediction_type="RawFormulaVal"),
            "curves": [np.asarray(v) for part in curves.values() for v in part.values()]}


def work(case):
    n, F, T, D = case["rows"], case["cols"], case["trees"], case["depth"]
    dims = {"MultiClass": 5}.get(case.get("loss"), case.get("dims", 1))
    if case["kind"] == "fit":
        cols = F + case["cats"]
        # the table and the target once; for every tree each document's bins (one byte a column), its cursor and its
        # target once, and its cursor written
        return {"bytes": float(n * (4 * cols + 4) + T * n * (cols + 8 * dims + 4)),
                "flops": float(T) * D * n * (F + case["cats"]) * (dims + 1) / 2.0}
    return {"bytes": float(n * (4 * min(F, T * D) + 4 * dims)), "flops": float(n) * T * (D + dims)}


def tolerance(case):
    if case["kind"] != "fit":
        # fp32 sums of 200 to 1000 leaf values against 64-bit sums and against the reverse order: 2e-7 to 8e-7, largest
        # difference of a value 1.2e-6 to 4.7e-6 of the root mean square
        return {"rel": 3e-6, "max": 2e-5}
    # Which split is the best is a comparison: where two candidates are equal to within the rounding of fp32 sums, another
    # order of the same sums can pick the other one, and the trees after it follow.  Measured on 55 pairs of runs (the same
    # code twice, and histograms summed in 13 to 16 against 24 bits a document): 53 pairs agree to 3e-5, two have one tree
    # that differs, which moves the predictions by 0.010 and 0.017 and leaves the loss curve alone to 1e-4.
    return {"rel": 0.03, "max": 0.9}


def exact(case, seed):
    """The sum of the leaves in 64 bits; a whole fit has no such value."""
    if case["kind"] == "fit":
        return None
    grid, feat, pick, vals = _trees(case, seed)
    columns = _rows(case, seed).t().contiguous()
    vals = torch.from_numpy(vals).cuda().view(case["trees"], 1 << case["depth"], case["dims"])
    out = torch.full((case["rows"], case["dims"]), 0.1, dtype=torch.float64, device="cuda")
    for t in range(case["trees"]):
        leaf = torch.zeros(case["rows"], dtype=torch.int64, device="cuda")
        for d in range(case["depth"]):
            j = int(feat[t, d])
            leaf |= (columns[j] > float(grid[j, pick[t, d]])).long() << d
        out += vals[t][leaf]
    if case["kind"] == "score":
        return out.t().contiguous()
    return (out[:, 0] if case["dims"] == 1 else out).cpu().numpy()
