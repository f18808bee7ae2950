"""The work a user of this framework has it do, as cases that can be timed.

Five kinds of calls, each through the package's public entry points:

  fit      a whole fit on a binned plane: booster, rounds, trees and training
           scores back on the host
  many     many independent fits in flight together
  predict  an ensemble's scores of a batch of raw rows (a request plane
           refilled, then the plan): host rows for requests, device rows for
           bulk scoring
  shap     TreeSHAP contributions of a batch, the same way
  cuts     cut fitting over a raw matrix in device memory

Inputs are seeded draws on the GPU, of the shapes and distributions of the
benchmark's workloads (bonsai_b200/synth.py): Friedman-like small regression,
tall binary, wide sparse, one-hot multiclass, ragged regression datasets, and
a 1,000-tree ensemble to serve.
"""

from __future__ import annotations

import math

import numpy as np
import torch

import bonsai_b200 as bb

LEAF = 0xFFFFFFFF
DEV = "cuda"


# ---- the cases ----------------------------------------------------------------

def _fit(name, data, rows, features, rounds, mode, **kw):
    case = dict(name=name, kind="fit", data=data, rows=rows, features=features, rounds=rounds,
                mode=mode, objective="mse", grower="depthwise", max_depth=6, max_leaves=31,
                n_classes=0, max_bin=255, subsample=1.0, feature_fraction=1.0, weighted=False)
    case.update(kw)
    return case


def _serve(name, kind, rows, features=28, trees=1000, depth=8, on_device=False):
    return dict(name=name, kind=kind, rows=rows, features=features, trees=trees, depth=depth,
                on_device=on_device)


def listed():
    return [
        # the everyday small regression in the default (exact) form: launch latency
        _fit("fit_small_exact", "regression", 20_640, 8, 100, "exact"),
        # the headline workload: a tall click/physics table, quantised gradients
        _fit("fit_tall_int8", "tall", 10_000_000, 28, 200, "int8", objective="logloss",
             max_depth=8),
        # the same table in the exact form, whose trees equal the CPU grower's
        _fit("fit_tall_exact", "tall", 10_000_000, 28, 20, "exact", objective="logloss",
             max_depth=8),
        # a wide sparse feature store: leafwise trees, row sample per tree
        _fit("fit_wide_leafwise", "wide", 1_000_000, 2_000, 25, "int8", grower="leafwise",
             max_depth=255, max_leaves=255, max_bin=256, subsample=0.8),
        # seven classes over continuous and one-hot columns, oblivious trees
        _fit("fit_multiclass", "onehot", 581_012, 54, 50, "int8", objective="softmax",
             grower="levelwise", max_depth=8, n_classes=7),
        # one model per store / fold: 64 uneven datasets in flight together
        dict(name="fit_many", kind="many", sets=64, features=28, rounds=100, mode="int8",
             max_depth=6, rows_lo=1_000, rows_hi=200_000),
        # one online request
        _serve("predict_1", "predict", 1),
        # a ragged micro-batch of requests
        _serve("predict_10k", "predict", 10_007),
        # bulk scoring of a table that is already on the GPU
        _serve("predict_1m", "predict", 1_000_000, on_device=True),
        # explanations for a page of requests
        _serve("shap_100", "shap", 100),
        # explanations for a whole table
        _serve("shap_100k", "shap", 100_000, on_device=True),
        # cuts for a tall table (a 200,000-row sample of it, as the mappers take)
        dict(name="cuts_tall", kind="cuts", rows=4_000_000, features=28, max_bin=255),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _rounds(rng, per_round_s):
    """5 to 100 rounds, about half a second in all at most."""
    most = max(5, min(100, int(0.5 / per_round_s)))
    return rng.randint(max(5, most // 2), most)


def draw(rng):
    kind = rng.choice(["fit"] * 10 + ["many", "cuts"] + ["predict"] * 4 + ["shap"] * 4)
    if kind == "predict":
        rows = _log(rng, 1, 1_000_000)
        return {k: v for k, v in _serve("", "predict", rows, rng.choice([8, 13, 28, 54]),
                                        _log(rng, 100, 1000), rng.randint(4, 8),
                                        rows > 100_000).items() if k != "name"}
    if kind == "shap":
        rows = _log(rng, 1, 50_000)
        return {k: v for k, v in _serve("", "shap", rows, rng.choice([8, 13, 28, 54]),
                                        _log(rng, 100, 1000), rng.randint(4, 8),
                                        rows > 10_000).items() if k != "name"}
    if kind == "cuts":
        return dict(kind="cuts", rows=_log(rng, 5_000, 4_000_000),
                    features=rng.choice([8, 28, 54, 131]), max_bin=rng.choice([63, 255, 256]))
    if kind == "many":
        return dict(kind="many", sets=rng.randint(8, 48), features=rng.choice([13, 28]),
                    rounds=rng.randint(20, 60), mode=rng.choice(["int8", "int8", "exact"]),
                    max_depth=rng.randint(4, 7), rows_lo=1_000, rows_hi=100_000)
    mode = rng.choice(["int8", "int8", "exact", "exact", "int16"])
    per = 9e-11 if mode == "exact" else 6e-12  # seconds per (row, feature) of a round, about
    data = rng.choice(["regression", "tall", "tall", "onehot", "wide"])
    kw = dict(max_depth=rng.randint(4, 8), weighted=rng.random() < 0.2,
              feature_fraction=rng.choice([1.0, 1.0, 1.0, 0.8]))
    grower = rng.choice(["depthwise", "depthwise", "levelwise", "leafwise"])
    if data == "regression":
        rows, features = _log(rng, 1_000, 500_000), 8
        kw["objective"] = rng.choice(["mse", "mse", "poisson"])
    elif data == "tall":
        rows, features = _log(rng, 20_000, 8_000_000), 28
        kw["objective"] = "logloss"
        grower = "depthwise" if rows > 2_000_000 else grower
    elif data == "onehot":
        rows, features = _log(rng, 20_000, 600_000), 54
        kw.update(objective="softmax", n_classes=7)
        grower = rng.choice(["levelwise", "depthwise"])
    else:
        features = rng.choice([100, 333, 1000, 2000])
        rows = min(_log(rng, 10_000, 800_000), (40_000_000 if mode == "exact"
                                                else 1_600_000_000) // features)
    if rows <= 1_000_000:
        kw["subsample"] = rng.choice([1.0, 1.0, 0.8])
    if grower == "leafwise":
        kw.update(max_depth=255, max_leaves=rng.choice([31, 63, 255]))
    trees = kw.get("n_classes", 0) or 1
    one = trees * (2e-3 + rows * features * per) + (8e-3 if grower == "leafwise" else 0.0)
    case = _fit("", data, rows, features, _rounds(rng, one), mode, grower=grower, **kw)
    del case["name"]
    return case


# ---- inputs -------------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device=DEV)


def _step_values(X, g, n_trees=8):
    """Sum of n_trees random depth-4 step trees over X's columns."""
    n, F = X.shape
    y = torch.zeros(n, device=DEV)
    for _ in range(n_trees):
        feats = torch.randint(0, F, (15,), generator=g, device=DEV)
        thr = _randn(g, 15)
        leaves = _randn(g, 16)
        idx = torch.zeros(n, dtype=torch.int64, device=DEV)
        for _ in range(4):
            x = X.gather(1, feats[idx][:, None])[:, 0]
            idx = 2 * idx + 1 + (x > thr[idx])
        y += leaves[idx - 15]
    return y


def _table(data, n, F, seed, n_classes, objective):
    """(X on the GPU, labels on the host) of one of the data families."""
    g = _gen(seed)
    if data == "regression":
        X = _randn(g, n, F)
        X[:, 0::2] = torch.rand(n, (F + 1) // 2, generator=g, device=DEV)
        X[:, 1::2] = X[:, 1::2].exp()
        y = (torch.sin(3.0 * X[:, 0]) + X[:, 1] * X[:, 2] + 0.5 * torch.log1p(X[:, 3])
             + 0.1 * _randn(g, n))
        if objective == "poisson":
            y = torch.poisson(y.clamp(0.05, 20.0), generator=g)
    elif data == "tall":
        X = torch.empty(n, F, device=DEV)
        B = _randn(g, n, 21)
        X[:, :21] = B
        X[:, 21] = B[:, 0] * B[:, 1]
        X[:, 22] = B[:, 2].abs()
        X[:, 23] = B[:, 3] * B[:, 4]
        X[:, 24] = (B[:, 5] * B[:, 6]).abs()
        X[:, 25] = B[:, 7] * B[:, 8]
        X[:, 26] = B[:, 9].abs()
        X[:, 27] = B[:, 10] * B[:, 11]
        w = 0.5 * _randn(g, F)
        p = torch.sigmoid((X * w).sum(1) + 0.5 * B[:, 0] * B[:, 1])
        y = (torch.rand(n, generator=g, device=DEV) < p).float()
    elif data == "wide":
        X = torch.empty(n, F, device=DEV)
        y = torch.empty(n, device=DEV)
        terms = [torch.randperm(F, generator=g, device=DEV)[:2 + k % 2] for k in range(20)]
        for s in range(0, n, 65_536):
            e = min(n, s + 65_536)
            Xc = _randn(g, e - s, F).exp_()
            gone = torch.rand(e - s, F, generator=g, device=DEV) < 0.9
            Z = Xc.masked_fill(gone, 0.0)
            y[s:e] = sum(Z[:, t].prod(1) for t in terms) + 0.1 * _randn(g, e - s)
            X[s:e] = Xc.masked_fill_(gone, float("nan"))
    else:  # 10 continuous columns, one-hot blocks of 4 and 40
        c = _randn(g, n, 10)
        W = _randn(g, 10, n_classes)
        logits = (c[:, :, None] * W).sum(1) + 0.5 * c[:, :n_classes] * c[:, 1:n_classes + 1]
        a = (logits.argmax(1) + torch.randint(0, 2, (n,), generator=g, device=DEV)) % 4
        b = (logits.flip(1).argmax(1) * 5
             + torch.randint(0, 6, (n,), generator=g, device=DEV)) % 40
        X = torch.zeros(n, F, device=DEV)
        X[:, :10] = c
        X[torch.arange(n, device=DEV), 10 + a] = 1.0
        X[torch.arange(n, device=DEV), 14 + b] = 1.0
        bump = 0.5 * _randn(g, 44, n_classes)
        y = (logits + bump[a] + bump[4 + b]).argmax(1).float()
    return X, y.cpu().numpy()


def _quantile_cuts(S, max_bin=255):
    """The quantile-stride cuts of S's columns (distinct continuous values)."""
    n, F = S.shape
    step = max(-(-n // (max_bin - 1)), 1)
    V = S.sort(dim=0).values[step::step].T.cpu().numpy()
    cuts, off = [], [0]
    for col in V:
        c = np.concatenate([np.unique(col), [np.finfo(np.float32).max, np.inf]])
        cuts.append(c.astype(np.float32))
        off.append(off[-1] + len(c))
    return np.concatenate(cuts), np.asarray(off, np.uint32)


def _codes(X, cuts, off):
    """Bin codes [rows, features]: cuts below the value; NaN is the last bin."""
    out = torch.empty(X.shape, dtype=torch.int64, device=DEV)
    for f in range(X.shape[1]):
        c = torch.as_tensor(cuts[off[f]:off[f + 1]], device=DEV)
        x = X[:, f].contiguous()
        out[:, f] = torch.where(x.isnan(), len(c) - 1, torch.searchsorted(c, x))
    return out


def _ensemble(case, seed):
    """An ensemble as a boosted fit leaves it: depth-limited trees split at bin
    borders, some features far more often than others, nodes of fewer than 40
    of the 20,000 fit rows left as leaves, covers from those rows, the leaf
    values shrinking over the rounds. Returns the trees as heaps [T, 2^(D+1) - 1]
    on the GPU, and the cuts."""
    T, D, F = case["trees"], case["depth"], case["features"]
    g = _gen(seed)
    S = _randn(g, 20_000, F)
    cuts, off = _quantile_cuts(S)
    codes = _codes(S, cuts, off)
    last = torch.as_tensor(np.diff(off.astype(np.int64)) - 1, device=DEV)
    m = 2 ** (D + 1) - 1
    weight = torch.rand(F, generator=g, device=DEV) ** 2 + 0.02
    feat = torch.multinomial(weight, T * m, replacement=True, generator=g).reshape(T, m)
    u = (0.5 + 0.22 * _randn(g, T, m)).clamp(0.02, 0.97)
    split = (u * last[feat]).long().clamp(max=250)
    default_left = torch.randint(0, 2, (T, m), generator=g, device=DEV)
    at = torch.zeros(T, 20_000, dtype=torch.int64, device=DEV)
    cover = torch.zeros(T, m, device=DEV)
    rows = torch.arange(20_000, device=DEV)[None, :]
    one = torch.ones(T, 20_000, device=DEV)
    for d in range(D + 1):
        cover.scatter_add_(1, at, one)
        if d < D:
            f = feat.gather(1, at)
            right = codes[rows, f] > split.gather(1, at)
            at = 2 * at + 1 + right
    parent = (torch.arange(1, m, device=DEV) - 1) // 2
    inner = torch.zeros(T, m, dtype=torch.bool, device=DEV)
    first = 2 ** D - 1
    both = torch.minimum(cover[:, 1::2], cover[:, 2::2])
    inner[:, :first] = (both >= 20) & (cover[:, :first] >= 40)
    live = torch.ones(T, m, dtype=torch.bool, device=DEV)
    for d in range(1, D + 1):
        lv = slice(2 ** d - 1, 2 ** (d + 1) - 1)
        up = parent[2 ** d - 2:2 ** (d + 1) - 2]
        live[:, lv] = live[:, up] & inner[:, up]
    inner &= live
    shrink = torch.exp(-3.0 * torch.arange(T, device=DEV) / T)[:, None]
    value = torch.where(inner, 0.0, _randn(g, T, m) * shrink)
    return dict(feat=feat, split=split, default_left=default_left, cover=cover, inner=inner,
                live=live, value=value), cuts, off


def _trees(E, cuts, off):
    """The heaps as the package's trees (breadth-first node tables)."""
    H = {k: v.cpu().numpy() for k, v in E.items()}
    T, m = H["feat"].shape
    ids = np.cumsum(H["live"], axis=1) - 1
    out = []
    for t in range(T):
        at = np.flatnonzero(H["live"][t])
        inner = H["inner"][t, at]
        child = np.where(inner, 2 * at + 1, 0)
        left = np.where(inner, ids[t, child], 0).astype(np.uint32)
        f, s = H["feat"][t, at], H["split"][t, at]
        value = np.where(inner, cuts[off[f].astype(np.int64) + s], H["value"][t, at])
        out.append(bb.Tree(
            feature=np.where(inner, f, LEAF).astype(np.uint32),
            value=value.astype(np.float32), left=left,
            right=np.where(inner, left + 1, 0).astype(np.uint32),
            default_left=np.where(inner, H["default_left"][t, at], 0).astype(np.uint8),
            gains=inner.astype(np.float32), covers=H["cover"][t, at].astype(np.float32),
            split_bin=np.where(inner, s, 0).astype(np.uint32),
            depth=int(np.floor(np.log2(at.max() + 1))), n_leaves=int((~inner).sum())))
    return out


def _requests(case, seed):
    """Raw request rows: N(0, 1), 2% of the values missing."""
    g = _gen(seed + 77)
    X = _randn(g, case["rows"], case["features"])
    X[torch.rand(X.shape, generator=g, device=DEV) < 0.02] = float("nan")
    return X


INIT, RATE = 0.25, 0.1


def _params(case, objective="mse", grower="depthwise"):
    kw = {k: case[k] for k in ("max_depth", "max_leaves", "n_classes", "subsample",
                               "feature_fraction") if k in case}
    return bb.TrainParams(objective=objective, grower=grower, hist_mode=case["mode"],
                          learning_rate=0.1, min_data_in_leaf=20, seed=1, use_graph=True, **kw)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "fit":
        X, y = _table(case["data"], case["rows"], case["features"], seed, case["n_classes"],
                      case["objective"])
        cuts, off = bb.fit_cuts_device(X, max_bin=case["max_bin"])
        plane = bb.Plane.from_device(X, cuts, off)
        w = None
        if case["weighted"]:
            w = np.random.default_rng(seed).uniform(0.5, 2.0, len(y)).astype(np.float32)
        return dict(kind=kind, plane=plane, y=y, weights=w, rounds=case["rounds"],
                    params=_params(case, case["objective"], case["grower"]))
    if kind == "many":
        g = _gen(seed)
        planes, ys = [], []
        for k in range(case["sets"]):
            # the sizes spread evenly over the range's logarithm
            u = (k * 29 % case["sets"] + 0.5) / case["sets"]
            n = int(case["rows_lo"] * (case["rows_hi"] / case["rows_lo"]) ** u)
            X = _randn(g, n, case["features"])
            y = _step_values(X, g) + 0.1 * _randn(g, n)
            cuts, off = _quantile_cuts(X)
            planes.append(bb.Plane.from_device(X, cuts, off))
            ys.append(y.cpu().numpy())
        return dict(kind=kind, planes=planes, ys=ys, rounds=case["rounds"],
                    params=_params(case))
    if kind == "cuts":
        return dict(kind=kind, X=_randn(_gen(seed), case["rows"], case["features"]),
                    max_bin=case["max_bin"])
    E, cuts, off = _ensemble(case, seed)
    trees = _trees(E, cuts, off)
    X = _requests(case, seed)
    some = bb.Plane.from_device(X[:1].contiguous(), cuts, off)
    plan = (bb.PredictPlan if kind == "predict" else bb.ShapPlan)(some, trees, INIT, RATE)
    request = bb.Plane.like(some, case["rows"])
    state = dict(kind=kind, plan=plan, request=request, on_device=case["on_device"])
    if case["on_device"]:
        state["X"] = X
        shape = (case["rows"],) if kind == "predict" else (case["rows"], case["features"] + 1)
        state["out"] = torch.empty(shape, device=DEV, dtype=torch.float32 if kind == "predict"
                                   else torch.float64)
    else:
        state["X"] = X.cpu().numpy()
    return state


# ---- one pass -----------------------------------------------------------------

def _tables(trees, params):
    """A fit's trees as arrays [trees, nodes], short trees filled up with zeros."""
    room = 4 * params.max_leaves if params.grower == "leafwise" else 2 ** (params.max_depth + 1)
    out = {}
    for k in ("feature", "value", "left", "right", "default_left", "gains", "covers",
              "split_bin"):
        a = out[k] = np.zeros((len(trees), room), getattr(trees[0], k).dtype)
        for row, t in zip(a, trees):
            v = getattr(t, k)
            row[:len(v)] = v
    return out


def run(state):
    kind = state["kind"]
    if kind == "fit":
        b = bb.Booster(state["plane"], state["y"], state["params"], max_trees=state["rounds"],
                       weights=state["weights"])
        b.update(state["rounds"])
        trees, scores = b.trees(), b.scores()
        b.close()
        return dict(trees=_tables(trees, state["params"]), scores=scores)
    if kind == "many":
        fits = [bb.Booster(p, y, state["params"], max_trees=state["rounds"])
                for p, y in zip(state["planes"], state["ys"])]
        for b in fits:
            b.update(state["rounds"], sync=False)
        for b in fits:
            b.sync()
        trees = [t for b in fits for t in b.trees()]
        scores = np.concatenate([b.scores() for b in fits])
        for b in fits:
            b.close()
        return dict(trees=_tables(trees, state["params"]), scores=scores)
    if kind == "cuts":
        return bb.fit_cuts_device(state["X"], max_bin=state["max_bin"])
    plan, request = state["plan"], state["request"]
    request.refill(state["X"], x_on_device=state["on_device"])
    if not state["on_device"]:
        return plan.run(request)
    plan.launch(request, state["out"].data_ptr(), torch.cuda.current_stream().cuda_stream)
    return state["out"]


# ---- what a pass cannot do without --------------------------------------------

def work(case):
    kind = case["kind"]
    if kind == "fit":
        n, F = case["rows"], case["features"]
        trees = case["rounds"] * max(1, case["n_classes"])
        leaves = case["max_leaves"] if case["grower"] == "leafwise" else 2 ** case["max_depth"]
        nodes = min(2 * leaves, 2 * n // 20 + 1)
        # each tree reads every (sampled) row's codes, label and score and
        # writes the score; two adds per (row, feature)
        rows = n * case["subsample"]
        return dict(bytes=trees * (rows * F * case["feature_fraction"] + 12.0 * n + 29.0 * nodes),
                    flops=trees * 2.0 * rows * F * case["feature_fraction"])
    if kind == "many":
        lo, hi = case["rows_lo"], case["rows_hi"]
        n = case["sets"] * (hi - lo) / math.log(hi / lo)  # sizes spread over the logarithm
        per = n * (case["features"] + 12.0) + case["sets"] * 29.0 * 2 ** (case["max_depth"] + 1)
        return dict(bytes=case["rounds"] * per, flops=case["rounds"] * 2.0 * n * case["features"])
    if kind == "cuts":
        n = min(case["rows"], 200_000)
        return dict(bytes=4.0 * case["features"] * (n + case["max_bin"]),
                    flops=float(n * case["features"] * math.log2(max(2, n))))
    n, F, T, D = case["rows"], case["features"], case["trees"], case["depth"]
    leaves = T * 2 ** D
    if kind == "predict":
        return dict(bytes=4.0 * n * (F + 1) + 8.0 * leaves, flops=2.0 * n * T * D)
    # each leaf path's D elements at D/2 Gauss points, prefix and suffix
    # products and sums
    return dict(bytes=4.0 * n * F + 8.0 * n * (F + 1) + 16.0 * D * leaves,
                flops=float(n) * leaves * D * max(1, D // 2) * 4)


# ---- the same results in 64 bits ----------------------------------------------

def _paths(E, last):
    """Every leaf's path over all trees: per step its feature, the cover
    fraction of the side taken, split bin, side and default direction."""
    T, m = E["feat"].shape
    t, at = torch.nonzero(E["live"] & ~E["inner"], as_tuple=True)
    steps = []
    node = at
    for _ in range(int(math.log2(m + 1)) - 1):
        up = torch.where(node > 0, (node - 1) // 2, 0)
        real = node > 0
        cov = E["cover"].double()
        frac = torch.where(real, cov[t, node] / cov[t, up], 1.0)
        steps.append((E["feat"][t, up], E["split"][t, up], E["default_left"][t, up] == 1,
                      node % 2 == 1, real, frac))
        node = up
    return t, at, [torch.stack(s, 1) for s in zip(*steps)]


def exact(case, seed):
    kind = case["kind"]
    if kind == "cuts":
        X = _randn(_gen(seed), case["rows"], case["features"])
        if case["rows"] > 200_000:
            pick = np.random.Generator(np.random.PCG64(0)).choice(case["rows"], size=200_000,
                                                                  replace=False)
            X = X[torch.as_tensor(np.sort(pick), device=DEV)]
        return _quantile_cuts(X, case["max_bin"])
    if kind not in ("predict", "shap"):
        return None  # a tree's splits are choices: no 64-bit value stands beside them
    E, cuts, off = _ensemble(case, seed)
    codes = _codes(_requests(case, seed), cuts, off)
    last = torch.as_tensor(np.diff(off.astype(np.int64)) - 1, device=DEV)
    n, F = codes.shape
    rate, init = float(np.float32(RATE)), float(np.float32(INIT))
    if kind == "predict":
        total = torch.zeros(n, dtype=torch.float64, device=DEV)
        rows = torch.arange(n, device=DEV)
        for t in range(case["trees"]):
            at = torch.zeros(n, dtype=torch.int64, device=DEV)
            for _ in range(case["depth"]):
                f = E["feat"][t][at]
                c = codes[rows, f]
                left = torch.where(c == last[f], E["default_left"][t][at] == 1,
                                   c <= E["split"][t][at])
                at = torch.where(E["inner"][t][at], 2 * at + 2 - left.long(), at)
            total += E["value"][t][at].double()
        return init + rate * total
    t, leaf, (feat, split, dleft, is_left, real, frac) = _paths(E, last)
    if n * len(t) > 60_000_000:
        return None
    K = feat.shape[1]
    value = E["value"][t, leaf].double()
    x, w = np.polynomial.legendre.leggauss(max(1, (K + 1) // 2))
    x = torch.as_tensor(0.5 * (x + 1.0), device=DEV)
    w = torch.as_tensor(0.5 * w, device=DEV)
    # a feature's steps merge into its first one: fractions multiply, every
    # condition has to hold; the others become elements that change nothing
    same = (feat[:, :, None] == feat[:, None, :]) & real[:, :, None] & real[:, None, :]
    head = real & ~(same & torch.ones(K, K, dtype=torch.bool, device=DEV).tril(-1)).any(2)
    z = torch.where(same, frac[:, None, :], 1.0).prod(2)
    z = torch.where(head, z, 1.0)
    phi = torch.zeros(n, F + 1, dtype=torch.float64, device=DEV)
    for s in range(0, len(t), 4096):
        e = slice(s, s + 4096)
        for r in range(0, n, 256):
            c = codes[r:r + 256][:, feat[e]]
            goes_left = torch.where(c == last[feat[e]], dleft[e], c <= split[e])
            ok = (goes_left == is_left[e]) | ~real[e]
            miss = (same[e].double() * (~ok).double()[:, :, None, :]).sum(3) > 0
            one = torch.where(head[e], (~miss).double(), 1.0)
            dz = one - z[e]
            into = torch.zeros_like(dz)
            for p in range(len(x)):
                fac = z[e] + dz * x[p]
                before = torch.ones_like(fac)
                after = torch.ones_like(fac)
                for k in range(1, K):
                    before[:, :, k] = before[:, :, k - 1] * fac[:, :, k - 1]
                    after[:, :, K - 1 - k] = after[:, :, K - k] * fac[:, :, K - k]
                into += w[p] * before * after
            into = (into * dz * value[e][:, None]).reshape(c.shape[0], -1)
            phi[r:r + 256].index_add_(1, feat[e].reshape(-1), into)
    # the bias: every tree's cover-weighted mean leaf
    cover = E["cover"].double()
    bias = (value * frac.prod(1)).sum()
    phi[:, F] += bias
    phi *= rate
    phi[:, F] += init
    return phi
