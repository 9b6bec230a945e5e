"""What is timed of this framework: the calls a user's program makes, over the sizes it makes them at.

Six kinds of work, each through the package's public entry points:

  regress    ``LBRegressor(...).fit(X, y)``: squared error, a few rounds
  classify   ``LBClassifier(...).fit(X, y)``: log loss, binary (2 classes) or softmax
  tree       ``Tree(...).fit(X, g, h)``: one tree on the gradients of the user's own objective
  predict    ``LBRegressor.predict`` / ``LBClassifier.predict_proba`` of a fitted ensemble
  update     ``Tree.update(X, g, h)``: new leaf values for a tree that is kept
  histogram  ``stages.histogram``: one level's histograms, the stage that users time on its own

Inputs are synthetic and made on the GPU from the seed.  A matrix has continuous columns (uniform or
normal) and two columns of few distinct values (6 and 32), as tables in practice do.
"""
import math

import numpy as np
import torch

import legateboost_b200 as lb
from legateboost_b200 import stages

#: the fields of a case and their usual values
DEFAULTS = dict(rows=0, features=0, dtype="float32", outputs=1, depth=6, rounds=1, split_samples=256, feature_fraction=1.0,
                fixed_sketch=False, nodes=0, bins=256, floats=False)

#: rows an ensemble is grown on before it is asked for predictions (its cost, not what is timed)
GROW_ROWS = 20000


def _case(kind, **kw):
    return dict(DEFAULTS, kind=kind, **kw)


def listed():
    return [
        # A table of a few hundred rows, as in notebooks, tests and cross-validation folds: the time is
        # launches, allocations and host work.
        _case("regress", name="fit_small", rows=500, features=10, depth=4, rounds=10),
        # The regression example of the benchmark configurations: 200,000 x 50, depth 6.
        _case("regress", name="fit_200k", rows=200_000, features=50, depth=6, rounds=10),
        # A large single-GPU training job at depth 8 (the benchmark's `--workload train`).
        _case("regress", name="fit_10m", rows=10_000_000, features=64, depth=8, rounds=3),
        # Softmax over ten classes, 100 features (the multi-output configuration, at a fifth of its rows).
        _case("classify", name="fit_softmax10", rows=1_000_000, features=100, outputs=10, depth=8, rounds=3),
        # Binary classification in float64 on an odd shape with more than 256 split candidates per
        # feature (two-byte bins) and half of the features per tree.
        _case("classify", name="fit_binary_f64_fine", rows=300_003, features=37, dtype="float64", outputs=2, depth=7,
              rounds=3, split_samples=512, feature_fraction=0.5),
        # The largest: one deep tree on the gradients of the user's own loss, 100M x 64 (the scale-out
        # configuration on one GPU).
        _case("tree", name="tree_100m_depth10", rows=100_000_000, features=64, depth=10),
        # Serving: a handful of rows, where latency is what counts.
        _case("predict", name="predict_16_rows", rows=16, features=30, depth=6, rounds=100),
        # Batch scoring with a large ensemble (the ensemble-predict configuration, at a fifth of its rows).
        _case("predict", name="predict_10m", rows=10_000_000, features=100, depth=8, rounds=500),
        # Class probabilities of a ten-class model, a ragged number of rows.
        _case("predict", name="predict_proba10", rows=100_003, features=100, outputs=10, depth=8, rounds=50),
        # Scoring in float64.
        _case("predict", name="predict_f64", rows=1_000_000, features=64, dtype="float64", depth=8, rounds=100),
        # A kept tree on new gradients.
        _case("update", name="update_10m", rows=10_000_000, features=64, depth=8),
        # The histogram microbenchmark: 10M x 128 one-byte bins, the 128 nodes of level 7.
        _case("histogram", name="histogram_10m", rows=10_000_000, features=128, nodes=128),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(max(lo, hi))))))


def draw(rng):
    kind = rng.choice(["regress", "classify", "tree", "predict", "update", "histogram"])
    features = _log_int(rng, 4, 512)
    dtype = rng.choice(["float32", "float32", "float32", "float64"])
    size = 4 if dtype == "float32" else 8
    if kind == "histogram":
        features = _log_int(rng, 8, 256)
        bins, nodes = rng.choice([32, 100, 256, 256]), 2 ** rng.randint(0, 8)
        outputs = rng.choice([1, 1, 1, 2, 3])
        most = min(10_000_000, 1_280_000_000 // (features * outputs))
        return _case(kind, rows=_log_int(rng, 1000, most), features=features, outputs=outputs, nodes=nodes, bins=bins,
                     floats=rng.random() < 0.25)
    if kind == "update":
        outputs = rng.choice([1, 1, 1, 3])
        most = 2_560_000_000 // (features * size * outputs)
        return _case(kind, rows=_log_int(rng, 200, min(10_000_000, most)), features=features, dtype=dtype,
                     outputs=outputs, depth=rng.randint(3, 10))
    if kind == "predict":
        outputs, depth = rng.choice([1, 1, 1, 2, 3, 10]), rng.randint(3, 10)
        rounds = _log_int(rng, 1, 500 if outputs <= 2 else 100)
        most = min(4_000_000_000 // (features * size), 5_000_000_000 // (rounds * depth * (outputs if outputs > 2 else 1)))
        return _case(kind, rows=_log_int(rng, 1, min(10_000_000, most)), features=features, dtype=dtype,
                     outputs=outputs, depth=depth, rounds=rounds)
    split_samples = rng.choice([32, 100, 256, 256, 256, 256, 512, 2048])
    depth = rng.randint(3, 10)
    if kind == "tree":
        outputs, rounds = rng.choice([1, 1, 1, 2, 4]), 1
        cells = 25_600_000_000 // (size * outputs)  # no more than the largest listed matrix
    else:
        outputs, rounds = 1, rng.randint(1, 10)
        if kind == "classify":
            outputs = rng.choice([2, 2, 3, 10])
        cells = 2_560_000_000 // (size * rounds * (outputs if outputs > 2 else 1))
    if outputs > 1:
        features = min(features, 128)
    if split_samples > 256:
        # finer bins go with smaller tables: a level's histograms have features x outputs x bins entries
        features = min(features, 64)
        cells = min(cells, 100_000_000 // (rounds * outputs))
    fraction = rng.choice([1.0, 1.0, 1.0, 0.5])
    return _case(kind, rows=_log_int(rng, 100, min(100_000_000, cells // features)), features=features, dtype=dtype,
                 outputs=outputs, depth=depth, rounds=rounds, split_samples=split_samples, feature_fraction=fraction,
                 fixed_sketch=kind != "tree" and rng.random() < 0.2)


# ---- inputs ---------------------------------------------------------------------------------------
def _columns(case):
    """Columns of predictions: a binary classifier has one."""
    return 1 if case["kind"] == "classify" and case["outputs"] == 2 else case["outputs"]


def _generator(seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    return gen


def _matrix(gen, rows, features, dtype, normal):
    dt = torch.float32 if dtype == "float32" else torch.float64
    X = (torch.randn if normal else torch.rand)((rows, features), dtype=dt, device="cuda", generator=gen)
    X[:, 0] = torch.round(X[:, 0] * 5) / 5
    X[:, features // 2] = torch.round(X[:, features // 2] * 31) / 31
    return X


def _target(gen, X):
    """y = the sum of sin(6 x) over the first five columns, plus noise; float32."""
    y = 0.1 * torch.randn(X.shape[0], dtype=torch.float32, device="cuda", generator=gen)
    for j in range(min(5, X.shape[1])):
        y += torch.sin(6 * X[:, j]).to(torch.float32)
    return y


def _labels(gen, X, classes):
    """argmax of X[:, :10] W plus noise; every class occurs."""
    m = min(10, X.shape[1])
    W = torch.randn((m, classes), dtype=X.dtype, device="cuda", generator=gen)
    z = X[:, :m] @ W + 0.5 * torch.randn((X.shape[0], classes), dtype=X.dtype, device="cuda", generator=gen)
    y = z.argmax(dim=1)
    y[:classes] = torch.arange(classes, device="cuda")[: y.shape[0]]
    return y


def _base(case):
    return lb.Tree(max_depth=case["depth"], split_samples=case["split_samples"], feature_fraction=case["feature_fraction"])


def _estimator(case, seed):
    kind = lb.LBClassifier if case["kind"] == "classify" or case["outputs"] > 1 else lb.LBRegressor
    return kind(n_estimators=case["rounds"], base_models=(_base(case),), random_state=seed, fixed_sketch=case["fixed_sketch"])


def _gradients(gen, rows, outputs):
    """What a loss of the user's own gives: residuals times a learning rate, weights around one."""
    g = torch.randn((rows, outputs), dtype=torch.float64, device="cuda", generator=gen).mul_(0.1)
    h = torch.rand((rows, outputs), dtype=torch.float64, device="cuda", generator=gen).add_(0.5)
    return g, h


def prepare(case, seed):
    gen = _generator(seed)
    kind, rows, features = case["kind"], case["rows"], case["features"]
    if kind == "histogram":
        return _prepare_histogram(case, gen, seed)
    if kind == "predict":
        many = _matrix(gen, GROW_ROWS, features, case["dtype"], False)
        y = _target(gen, many) if case["outputs"] == 1 else _labels(gen, many, case["outputs"])
        model = _estimator(case, seed).fit(many, y)
        return dict(kind=kind, model=model, X=_matrix(gen, rows, features, case["dtype"], False), proba=case["outputs"] > 1)
    X = _matrix(gen, rows, features, case["dtype"], kind == "classify")
    if kind == "update":
        tree = _base(case).set_random_state(np.random.RandomState(seed))
        few = X[: min(rows, GROW_ROWS)].contiguous()
        signal = _target(gen, few).to(torch.float64)
        tree.fit(few, signal[:, None].repeat(1, case["outputs"]), torch.ones((few.shape[0], case["outputs"]), dtype=torch.float64, device="cuda"))
        g, h = _gradients(gen, rows, case["outputs"])
        return dict(kind=kind, tree=tree, X=X, g=g, h=h)
    if kind == "tree":
        g, h = _gradients(gen, rows, case["outputs"])
        g[:, 0] -= _target(gen, X)
        return dict(kind=kind, case=dict(case), seed=seed, X=X, g=g, h=h)
    y = _target(gen, X) if kind == "regress" else _labels(gen, X, case["outputs"])
    return dict(kind=kind, case=dict(case), seed=seed, X=X, y=y)


def _prepare_histogram(case, gen, seed):
    rows, F, K, nb, nodes = case["rows"], case["features"], case["outputs"], case["bins"], case["nodes"]
    bins = torch.zeros((rows, (F + 31) // 32 * 32), dtype=torch.uint8, device="cuda")
    bins[:, :F] = torch.randint(0, nb, (rows, F), dtype=torch.uint8, device="cuda", generator=gen)
    g = torch.randn((rows, K), dtype=torch.float64, device="cuda", generator=gen)
    h = torch.ones((rows, K), dtype=torch.float64, device="cuda")
    node = torch.randint(0, nodes, (rows,), dtype=torch.int32, device="cuda", generator=gen) + (nodes - 1)
    row_index, seg = stages.group_rows(node, nodes - 1, nodes)
    order, max_abs = row_index.long(), None
    if case["floats"]:
        pairs = torch.stack([g, h], dim=2).to(torch.float32)
    else:
        pairs, _, _, max_abs = stages.quantise(g, h, seed=seed, with_max_abs=True)
    row_ptr = torch.arange(F + 1, dtype=torch.int32, device="cuda") * nb
    kind = torch.float64 if case["floats"] else torch.int64
    return dict(kind="histogram", bins=bins, row_ptr=row_ptr, pairs=pairs[order].contiguous(), row_index=row_index, seg=seg,
                features=F, n_bins=nb, mode=1 if case["floats"] else 0, max_abs=max_abs,
                hist=torch.empty((nodes, K, F * nb, 2), dtype=kind, device="cuda"))


# ---- one pass -------------------------------------------------------------------------------------
def _arrays(tree):
    return [tree.feature, tree.split_value, tree.leaf_value, tree.gain, tree.hessian]


def run(state):
    kind = state["kind"]
    if kind == "histogram":
        return stages.histogram(state["bins"], state["row_ptr"], state["pairs"], state["row_index"], state["seg"],
                                state["features"], mode=state["mode"], hist=state["hist"], max_abs=state["max_abs"],
                                max_bins=state["n_bins"], total_bins=state["features"] * state["n_bins"],
                                pairs_by_position=True)
    if kind == "predict":
        return state["model"].predict_proba(state["X"]) if state["proba"] else state["model"].predict(state["X"])
    if kind == "update":
        tree = state["tree"].update(state["X"], state["g"], state["h"])
        return [tree.leaf_value, tree.hessian]
    if kind == "tree":
        tree = _base(state["case"]).set_random_state(np.random.RandomState(state["seed"]))
        return _arrays(tree.fit(state["X"], state["g"], state["h"]))
    model = _estimator(state["case"], state["seed"]).fit(state["X"], state["y"])
    return [model.model_init_] + [_arrays(t) for t in model]


# ---- what a pass cannot do without ----------------------------------------------------------------
def work(case):
    N, F, K, D, R = case["rows"], case["features"], _columns(case), case["depth"], case["rounds"]
    size = 4 if case["dtype"] == "float32" else 8
    kind, tree_nodes = case["kind"], 2 ** (D + 1) - 1
    if kind == "histogram":
        # a bin byte per cell, a pair of 8 bytes per row and output, a row id per row, the sums written
        return {"bytes": N * (F + 8 * K + 4) + case["nodes"] * K * F * case["bins"] * 16, "flops": 2 * N * F * K}
    if kind == "predict":
        K = 1 if case["outputs"] == 2 else K
        return {"bytes": N * (F * size + 8 * max(K, case["outputs"])) + R * tree_nodes * (12 + 8 * K), "flops": N * R * (D + K)}
    if kind == "update":
        return {"bytes": N * (F * size + 16 * K) + tree_nodes * (12 + 16 * K), "flops": N * (D + 2 * K)}
    tree_bytes = tree_nodes * (4 + 8 + 8 + 16 * K)
    per_row = 16 * K if kind == "tree" else (4 if kind == "regress" else 8)
    # two additions per row, feature, output and level for the histograms, of which the smaller child
    # of every pair has to be summed
    adds = 2 * N * F * K * (1 + 0.5 * (D - 1))
    return {"bytes": N * (F * size + per_row) + R * tree_bytes, "flops": R * adds}


def tolerance(case):
    kind = case["kind"]
    if kind == "histogram":
        return {"rel": 1e-5} if case["floats"] else "exact"
    if kind in ("predict", "update"):
        return {"rel": 1e-12, "max": 1e-9}  # float64 sums in another order
    # the splits follow from whole-number histograms; the values are float64
    return {"rel": 1e-9, "max": 1e-6, "differ": 0.0}
