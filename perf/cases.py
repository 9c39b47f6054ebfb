"""The prediction calls that users of `cuml_b200.fil.ForestInference` make, over the range of
forests and batches they make them with.

A case names a forest (how it was trained, trees, depth or leaves, features, outputs, precision),
a batch (rows, share of missing values, in device or host memory) and the call.  `listed()` are
typical points, `draw()` gives further ones of the same ranges.  Forest shapes are those of this
repository's benchmark configurations and of the usual defaults of tree libraries; forests and
rows are synthetic and made from the seed.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from cuml_b200.fil import ForestDesc, ForestInference, synthetic_complete_forest

# Limits of a drawn case, so that none costs more than the largest listed one: (row, tree, level)
# visits of forests of complete trees and of deep ragged ones, bytes of the batch, bytes of the
# outputs.
MOST_VISITS = {"boosted": 1.2e10, "classifier": 8e8, "regressor": 1.2e9}
MOST_INPUT = 1.5e9
MOST_OUTPUT = 4e8

BASE = {"forest": "boosted", "trees": 100, "depth": 6, "leaves": 0, "features": 32, "classes": 1,
        "categorical": 0, "missing": 0.0, "dtype": "float32", "rows": 1000,
        "memory": "device", "call": "predict_proba"}


def _case(name=None, **kw):
    case = dict(BASE, **kw)
    if name:
        case["name"] = name
    return case


def listed():
    return [
        # Online scoring: one row through the binary boosted forest of the headline benchmark.
        _case("one row", trees=1000, depth=8, features=256, rows=1),
        # A request of a scoring service: a small boosted forest, labels wanted.
        _case("small batch", trees=300, depth=6, features=50, rows=1000, call="predict"),
        # The same service with a micro-batch and the deep trees of an unpruned regression forest.
        _case("small batch, deep trees", forest="regressor", trees=100, depth=20, leaves=8000,
              features=30, rows=1024, call="predict"),
        # A notebook: a NumPy table through a random-forest classifier, result back as NumPy.
        _case("host table", forest="classifier", trees=100, depth=8, leaves=200, features=32,
              classes=2, rows=10_000, memory="host"),
        # A batch that is neither small nor large (20 k rows) on the headline forest.
        _case("medium batch", trees=1000, depth=8, features=256, rows=20_011),
        # A large NumPy array, bound for the GPU over the host link.
        _case("host array", trees=500, depth=6, features=128, rows=200_000, memory="host"),
        # Leaf indices as features for a second model: one output per row and tree.
        _case("leaf indices", trees=300, depth=6, features=60, rows=100_003, call="apply"),
        # Random-forest classifier of depth 8 over 32 features, a million rows.
        _case("classifier", forest="classifier", trees=100, depth=8, leaves=200, features=32,
              classes=2, rows=1_000_000),
        # Ten classes, categorical features, missing values, softmax.
        _case("multiclass, categorical, missing", trees=5000, depth=6, features=128, classes=10,
              categorical=8, missing=0.05, rows=150_000),
        # Unpruned regression forest in double precision.
        _case("deep regressor, double", forest="regressor", trees=200, depth=20, leaves=16_000,
              features=64, dtype="float64", rows=300_000, call="predict"),
        # The scale-out forest: trees of depth 10 over 512 features.
        _case("deep boosted", trees=2000, depth=10, features=512, rows=200_000),
        # Offline scoring on the headline forest.
        _case("large batch", trees=1000, depth=8, features=256, rows=1_500_000),
    ]


def _spread(rng, lo, hi):
    """A whole number between lo and hi, evenly spread over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    family = rng.choice(["boosted", "boosted", "boosted", "multiclass", "classifier", "regressor"])
    if family == "boosted":
        # from a small model of a tutorial to the scale-out forest
        case = _case(trees=_spread(rng, 50, 2000), depth=rng.randint(4, 10),
                     features=_spread(rng, 10, 512), missing=rng.choice([0.0, 0.0, 0.05]),
                     rows=_spread(rng, 1, 1_500_000),
                     call=rng.choice(["predict_proba", "predict_proba", "predict", "apply"]))
    elif family == "multiclass":
        classes = rng.randint(3, 10)
        case = _case(trees=classes * _spread(rng, 20, 500), depth=rng.randint(4, 8),
                     features=_spread(rng, 16, 128), classes=classes,
                     categorical=rng.choice([0, 4, 8]), missing=rng.choice([0.0, 0.05]),
                     rows=_spread(rng, 100, 300_000),
                     call=rng.choice(["predict_proba", "predict_proba", "predict"]))
    elif family == "classifier":
        case = _case(forest="classifier", trees=_spread(rng, 50, 300), depth=rng.randint(6, 10),
                     leaves=_spread(rng, 50, 400), features=_spread(rng, 8, 100),
                     classes=rng.randint(2, 6), rows=_spread(rng, 100, 1_000_000),
                     call=rng.choice(["predict_proba", "predict_proba", "predict"]))
    else:
        case = _case(forest="regressor", trees=_spread(rng, 50, 200), depth=rng.randint(14, 20),
                     leaves=_spread(rng, 4000, 16_000), features=_spread(rng, 10, 64),
                     dtype=rng.choice(["float32", "float64"]), rows=_spread(rng, 100, 300_000),
                     call=rng.choice(["predict", "predict", "apply"]))
    case["memory"] = rng.choice(["device", "device", "device", "host"])
    case["rows"] = max(1, min(case["rows"], _most_rows(case)))
    return case


def _sizes(case):
    """Bytes of a row, of a row's outputs, and of the forest's tests and leaves."""
    item = 8 if case["dtype"] == "float64" else 4
    row = case["features"] * item
    width = {"predict_proba": max(2, case["classes"]) * item, "apply": case["trees"] * 4,
             "predict": 4 if case["forest"] != "regressor" else item}[case["call"]]
    leaves = case["leaves"] or 1 << case["depth"]
    leaf = item * (case["classes"] if case["forest"] == "classifier" else 1)
    # a test is a feature, a threshold or category set, and a direction
    return row, width, case["trees"] * leaves * (leaf + item + 4)


def _most_rows(case):
    row, width, _ = _sizes(case)
    host = 0.1 if case["memory"] == "host" else 1.0  # the host link is slower
    return int(min(MOST_VISITS[case["forest"]] / (case["trees"] * case["depth"]),
                   MOST_INPUT * host / row, MOST_OUTPUT * host / width))


def _bagged_forest(case, g, device):
    """Trees as bagging grows them: every node splits its samples in a random proportion at the
    matching quantile of a normal feature, down to single samples or the depth limit, so that a
    row's path has the length it has in a fitted forest."""
    n_trees = case["trees"]
    tree = torch.arange(n_trees, device=device)
    count = torch.full((n_trees,), float(case["leaves"]), device=device, dtype=torch.float64)
    levels, total = [], 0
    for depth in range(case["depth"] + 1):
        n = int(tree.numel())
        share = 0.1 + 0.8 * torch.rand(n, generator=g, device=device, dtype=torch.float64)
        inner = (count >= 2) & (depth < case["depth"])
        n_left = torch.minimum(torch.clamp(torch.round(count * share), min=1), count - 1)
        rank = torch.cumsum(inner.to(torch.int64), 0) - 1
        first = torch.where(inner, total + n + 2 * rank, torch.full_like(rank, -1))
        levels.append({"tree": tree, "inner": inner, "left": first,
                       "threshold": math.sqrt(2.0) * torch.erfinv(2.0 * n_left / count - 1.0)})
        total += n
        tree = tree[inner].repeat_interleave(2)
        count = torch.stack([n_left[inner], (count - n_left)[inner]], 1).reshape(-1)
        if tree.numel() == 0:
            break
    flat = {k: torch.cat([lv[k] for lv in levels]) for k in levels[0]}
    # nodes of a tree go together, level by level
    order = torch.argsort(flat["tree"], stable=True)
    offsets = torch.zeros(n_trees + 1, dtype=torch.int64, device=device)
    offsets[1:] = torch.cumsum(torch.bincount(flat["tree"], minlength=n_trees), 0)
    place = torch.empty_like(order)
    place[order] = torch.arange(total, device=device)
    flat = {k: v[order] for k, v in flat.items()}
    inner = flat["inner"]
    left = torch.where(inner, place[flat["left"].clamp(min=0)] - offsets[flat["tree"]],
                       torch.full_like(place, -1)).to(torch.int32)
    threshold = torch.where(inner, flat["threshold"], torch.zeros_like(flat["threshold"]))
    if case["dtype"] == "float32":
        threshold = threshold.float().double()
    feature = torch.randint(0, case["features"], (total,), generator=g, device=device)
    k = case["classes"]
    if case["forest"] == "classifier":
        leaf = torch.rand((total, k), generator=g, device=device, dtype=torch.float64) ** 3 + 1e-3
        leaf = (leaf / leaf.sum(1, keepdim=True)).reshape(-1)
    else:
        leaf = torch.randn(total, generator=g, device=device, dtype=torch.float64)
    host = lambda t: t.cpu().numpy()  # noqa: E731
    return ForestDesc(
        n_features=case["features"], n_outputs=k, leaf_vector_len=k, tree_offsets=host(offsets),
        node_kind=host(inner.to(torch.uint8)), feature=host(torch.where(inner, feature, 0)),
        threshold=host(threshold), left=host(left), right=host(torch.where(inner, left + 1, -1)),
        default_left=np.zeros(total, np.uint8), leaf_value=host(leaf),
        average_tree_output=True, is_classifier=case["forest"] == "classifier",
        postproc="identity_multiclass" if case["forest"] == "classifier" else "identity",
        native_precision="double" if case["dtype"] == "float64" else "single")


def _rows(case, g, device):
    """Standard normal features; categorical ones hold categories, missing values are NaN."""
    dtype = getattr(torch, case["dtype"])
    x = torch.randn((case["rows"], case["features"]), generator=g, device=device, dtype=dtype)
    if case["categorical"]:
        shape = (case["rows"], case["categorical"])
        x[:, :case["categorical"]] = torch.randint(0, 32, shape, generator=g, device=device).to(dtype)
    if case["missing"]:
        x[torch.rand(x.shape, generator=g, device=device) < case["missing"]] = float("nan")
    return x


def prepare(case, seed):
    """The loaded model and the batch to predict."""
    device = torch.device("cuda:0")
    g = torch.Generator(device=device)
    g.manual_seed(seed)
    if case["forest"] == "boosted":
        desc = synthetic_complete_forest(
            case["trees"], case["depth"], case["features"], seed, n_classes=case["classes"],
            n_categorical=case["categorical"], n_categories=32)
    else:
        desc = _bagged_forest(case, g, device)
    model = ForestInference.load_from_treelite_model(
        desc, precision="double" if case["dtype"] == "float64" else "single")
    x = _rows(case, g, device)
    if case["memory"] == "host":
        x = x.cpu().numpy()
    return {"call": getattr(model, case["call"]), "x": x}


def run(state):
    return state["call"](state["x"])


def work(case):
    row, width, forest = _sizes(case)
    # one comparison per level of every tree, one addition per tree
    visits = case["trees"] * (min(case["depth"], 2 * math.log2(case["leaves"]))
                              if case["leaves"] else case["depth"])
    return {"bytes": case["rows"] * (row + width) + forest,
            "flops": case["rows"] * (visits + case["trees"])}


def tolerance(case):
    if case["call"] == "apply":
        return "exact"
    if case["forest"] != "regressor" and case["call"] == "predict":
        # labels: scores of different summation order may fall on either side of a tie
        return {"rel": 0.0, "differ": 1e-3}
    return {"rel": 1e-12} if case["dtype"] == "float64" else {"rel": 1e-5}
