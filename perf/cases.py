"""The work that users of this package have it do, as cases that can be timed and compared.

A case is one call of a public entry point on one set of inputs:

  kind "fit"      `fit(params, x_train=, y_train=, ...)`: quantile edges, upload, binarize, every boosting round, every
                  tree read back -- from ordinary (pageable) host arrays, as a user holds them -- and the training
                  predictions that boosting can be resumed from; with a validation set its metric is tracked
  kind "predict"  `m(x)` of a fitted model: upload, binarize, all trees, link, predictions back

The large sizes are the configurations of the package's own benchmark; the others are ordinary ones between them and the
smallest call (one row to score, a thousand rows to learn from).  Inputs are made on the GPU from the seed and brought to
the host: "uniform" and "normal" are the features of the benchmark configurations, "mixed" is what a table looks like --
uniform columns, long-tailed ones and small counts whose quantile edges coincide.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import __graft_entry__

pkg = __graft_entry__.load_package()

FIT = {"kind": "fit", "loss": "mse", "classes": 0, "data": "mixed", "dtype": "f32", "order": "F", "eta": 0.1, "rowsample": 1.0,
       "colsample": 1.0, "weights": False, "eval_rows": 0}
PREDICT = {"kind": "predict", "loss": "mse", "classes": 0, "data": "mixed", "dtype": "f32", "order": "C"}


def listed():
    fit = lambda name, **kw: {"name": name, **FIT, **kw}          # noqa: E731
    predict = lambda name, **kw: {"name": name, **PREDICT, **kw}  # noqa: E731
    return [
        # a first model on a small table, its validation loss tracked: latency and launches
        fit("fit_1503x7_logloss_eval", rows=1503, feats=7, depth=5, nbins=64, rounds=100, loss="logloss", dtype="f64", order="C", eval_rows=501),
        # benchmark configuration 1
        fit("fit_100k_x10", rows=100_000, feats=10, depth=6, nbins=32, rounds=200, data="uniform", dtype="f64"),
        # claim / visit counts: a log-link loss on an ordinary table, columns sampled, a numpy (row-major) array
        fit("fit_60k_x77_poisson", rows=60_013, feats=77, depth=6, nbins=64, rounds=50, loss="poisson", order="C", colsample=0.7),
        # weighted regression with a validation set, a numpy (row-major) array
        fit("fit_250k_x33_weighted_eval", rows=250_007, feats=33, depth=7, nbins=64, rounds=100, weights=True, eval_rows=50_021, order="C"),
        # benchmark configuration 2: row and column samples
        fit("fit_1M_x100_sampled", rows=1_000_000, feats=100, depth=6, nbins=64, rounds=200, data="uniform", dtype="f64", eta=0.05,
            rowsample=0.5, colsample=0.5),
        # benchmark configuration 4, a quarter of its rounds: five classes
        fit("fit_2M_x28_softmax", rows=2_000_000, feats=28, depth=8, nbins=64, rounds=50, loss="mlogloss", classes=5, data="normal"),
        # benchmark configuration 5: two-parameter likelihood
        fit("fit_5M_x50_gaussian", rows=5_000_000, feats=50, depth=7, nbins=32, rounds=200, loss="gaussian_mle", data="uniform"),
        # benchmark configuration 3, the headline
        fit("fit_10M_x100_deep", rows=10_000_000, feats=100, depth=11, nbins=64, rounds=200, data="uniform"),
        # scoring one row of a table, as a service does
        predict("predict_1_x10", rows=1, feats=10, depth=6, nbins=32, trees=100, dtype="f64"),
        # scoring a batch with a classifier
        predict("predict_20k_x28_softmax", rows=20_011, feats=28, depth=8, nbins=64, trees=200, loss="mlogloss", classes=5, data="normal"),
        # scoring a table with the headline's deep trees
        predict("predict_500k_x100_deep", rows=500_009, feats=100, depth=11, nbins=64, trees=200),
        # the inference half of benchmark configuration 5
        predict("predict_10M_x50_gaussian", rows=10_000_000, feats=50, depth=7, nbins=32, trees=200, loss="gaussian_mle", data="uniform", order="F"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _channels(loss, classes):
    """Gradient / hessian / weight sums that a histogram of the loss holds (mse: the hessian is twice the weight)."""
    return {"mse": 2, "mlogloss": 2 * classes + 1, "gaussian_mle": 5}.get(loss, 3)


def draw(rng):
    loss = rng.choice(("mse", "mse", "mse", "logloss", "poisson", "mlogloss", "gaussian_mle"))
    classes = rng.randint(3, 7) if loss == "mlogloss" else 0
    feats = _log_int(rng, 4, 128)
    nbins = rng.choice((32, 64, 64, 64, 128, 255))
    c = {"loss": loss, "classes": classes, "data": rng.choice(("mixed", "mixed", "uniform", "normal")), "dtype": rng.choice(("f32", "f32", "f64")),
         "order": rng.choice(("C", "F"))}
    if rng.random() < 0.4:
        rows = min(_log_int(rng, 1, 4_000_000), 200_000_000 // feats)
        return {**PREDICT, **c, "rows": rows, "feats": feats, "depth": rng.randint(4, 11), "nbins": nbins, "trees": _log_int(rng, 20, 200)}
    weights = rng.random() < 0.2
    exact = loss == "mse" and not weights
    depth = rng.randint(4, 9)
    rounds = _log_int(rng, 20, 200 if exact else 50)
    # no more work than a third of the headline's, no more input than a quarter of it
    most = 4e11 / (feats * rounds * (1 + (depth - 2) / 2) * (_channels(loss, classes) - 1))
    rows = min(_log_int(rng, 1000, 3_000_000), 250_000_000 // feats, int(most))
    depth = min(depth, int(math.log2(rows / 32)))  # no deeper than the rows carry
    return {**FIT, **c, "rows": rows, "feats": feats, "depth": depth, "nbins": nbins, "rounds": rounds, "eta": rng.choice((0.05, 0.1, 0.2)),
            "rowsample": rng.choice((1.0, 1.0, 0.5, 0.8)) if exact else 1.0, "colsample": rng.choice((1.0, 1.0, 0.5, 0.8)),
            "weights": weights, "eval_rows": rows // 4 if rng.random() < 0.3 else 0}


def _features(case, n, gen):
    """[n, feats] on the GPU, in the memory order of the case."""
    F, dt = case["feats"], torch.float32 if case["dtype"] == "f32" else torch.float64
    x = torch.empty((n, F) if case["order"] == "C" else (F, n), dtype=dt, device="cuda")
    if case["data"] == "uniform":
        x.uniform_(generator=gen)
    else:
        x.normal_(generator=gen)
    x = x if case["order"] == "C" else x.T
    if case["data"] == "mixed":
        x[:, 1::3] = torch.exp(x[:, 1::3])                              # long tails
        x[:, 2::3] = torch.floor(torch.abs(x[:, 2::3]) * 2.0)            # small counts
    return x


def _target(case, x, par, gen):
    """Target of `x` and row weights; `par` makes the parameters of the relation, the same for training and evaluation rows."""
    n, F = x.shape
    loss = case["loss"]
    if loss == "mlogloss":                       # argmax(x W + Gumbel(0, 1))
        W = torch.randn((F, case["classes"]), generator=par, device="cuda", dtype=x.dtype)
        u = torch.rand((n, case["classes"]), generator=gen, device="cuda")
        return torch.argmax(x @ W - torch.log(-torch.log(u * 0.999998 + 1e-6)), dim=1).cpu().numpy()
    beta = torch.randn(F, generator=par, device="cuda", dtype=x.dtype)
    s = (x @ beta).float()
    e = torch.randn(n, generator=gen, device="cuda")
    if loss == "mse":
        y = s + 0.1 * e
    elif loss == "gaussian_mle":
        y = s + torch.exp(0.5 * x[:, 0].float()) * e
    else:
        z = (s - s.mean()) / (s.std() + 1e-6)
        y = (z + 0.5 * e > 0).float() if loss == "logloss" else torch.poisson(torch.exp((0.6 * z).clamp(-4.0, 4.0)), generator=gen)
    return y.cpu().numpy()


def _host(x):
    """The same array on the host, memory order kept."""
    return x.cpu().numpy() if x.is_contiguous() else x.T.cpu().numpy().T


def _exact(case):
    """Integer sums of the gradients decide every split of least squares without weights: the trees are the same whatever
    the order of the additions."""
    return case["kind"] == "fit" and case["loss"] == "mse" and not case["weights"]


def _params(case, rounds):
    kw = dict(nrounds=rounds, max_depth=case["depth"], nbins=case["nbins"], eta=case.get("eta", 0.1), rowsample=case.get("rowsample", 1.0),
              colsample=case.get("colsample", 1.0))
    if case["loss"] == "mlogloss":
        return pkg.EvoTreeClassifier(**kw)
    if case["loss"] == "gaussian_mle":
        return pkg.EvoTreeMLE(**kw)
    return pkg.EvoTreeRegressor(loss=case["loss"], **kw)


def _model(case, gen, par):
    """A fitted model: full trees that least squares learns from a moderate table of the same distribution; the other losses
    take their splits and, for every output, their leaf values in another scale."""
    base = {**case, "loss": "mse"}
    xt = _features(case, 50_000 if case["depth"] > 8 else 20_000, gen)
    m = pkg.fit(_params(base, case["trees"]), x_train=_host(xt), y_train=_target(base, xt, par, gen))
    if case["loss"] == "mse":
        return m
    K = {"mlogloss": case["classes"], "gaussian_mle": 2}.get(case["loss"], 1)
    scale = np.float32(0.3 / max(np.abs(t.pred).max() for t in m.trees)) * np.random.default_rng(gen.initial_seed()).normal(size=K).astype(np.float32)
    trees = [pkg.Tree(t.feat, t.cond_bin, t.w, t.gain, np.ascontiguousarray(t.pred * scale), t.split) for t in m.trees]
    return pkg.EvoTree(case["loss"], K, trees, m.info)


def prepare(case, seed):
    gen = torch.Generator("cuda").manual_seed(seed)
    par = lambda: torch.Generator("cuda").manual_seed(seed + 1_000_003)  # noqa: E731
    if case["kind"] == "predict":
        return {"model": _model(case, gen, par()), "x": _host(_features(case, case["rows"], gen))}
    x = _features(case, case["rows"], gen)
    args = {"x_train": _host(x), "y_train": _target(case, x, par(), gen)}
    if case["weights"]:
        args["w_train"] = (0.25 + 2.0 * torch.rand(case["rows"], generator=gen, device="cuda")).cpu().numpy()
    del x
    if case["eval_rows"]:
        x = _features(case, case["eval_rows"], gen)
        args.update(x_eval=_host(x), y_eval=_target(case, x, par(), gen))
    return {"params": _params(case, case["rounds"]), "args": args, "exact": _exact(case)}


def run(state):
    if "model" in state:
        return {"pred": pkg.predict(state["model"], state["x"])}
    m, cache = pkg.fit(state["params"], return_cache=True, **state["args"])
    out = {"pred": cache.pred(), "bias": m.trees[0].pred, "edges": m.info["edges"]}
    cache.close()
    if m.info["logger"] is not None:
        out["metrics"] = np.array(m.info["logger"]["metrics"])
    if state["exact"]:
        out.update({"tree_" + k: np.concatenate([getattr(t, k) for t in m.trees]) for k in ("feat", "cond_bin", "split", "w", "gain", "pred")})
    return out


def work(case):
    n, F = case["rows"], case["feats"]
    es = 4 if case["dtype"] == "f32" else 8
    K = {"mlogloss": case["classes"], "gaussian_mle": 2}.get(case["loss"], 1)
    nodes = 2 ** case["depth"] - 1
    if case["kind"] == "predict":
        # features in, predictions out, the packed trees once; one comparison per tree and level
        return {"bytes": n * (F * es + 4 * K) + case["trees"] * nodes * (4 + 4 * K), "flops": n * case["trees"] * (case["depth"] - 1)}
    # the input once; per round every sampled row's bins and gradients at the root and half of them again at each further
    # level that is split (the other child is the difference), gradients written once; the trees
    ch = _channels(case["loss"], case["classes"])
    seen = case["rounds"] * n * case["rowsample"] * (1 + (case["depth"] - 2) / 2)
    Fs = math.ceil(case["colsample"] * F)
    return {"bytes": (n + case["eval_rows"]) * (F * es + 4 + 4 * case["weights"]) + seen * (Fs + 4 * (ch - 1)) + case["rounds"] * (n * 4 * (ch - 1) + nodes * (14 + 4 * K)),
            "flops": seen * Fs * ch}


def tolerance(case):
    if case["kind"] == "predict" or _exact(case):
        return {"rel": 1e-5, "max": 1e-4}          # sums of 32-bit leaf values; whole numbers are the same
    # The gradients of these losses are summed in 32 bits.  Two splits that separate the same rows, or nearly, tie to the last
    # bits of those sums, either is right, and the rounds after a tie differ: a change of eta by 2e-7 moves the training
    # predictions by 1e-7 in most cases of these ranges, by 1e-2 (one row: 0.3) in the deepest.  The trees of these
    # cases are not compared for that reason, what they add up to on every training row is.
    return {"rel": 2e-2, "max": 0.5}
