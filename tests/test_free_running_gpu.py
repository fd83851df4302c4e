"""Free-running fits against the oracle: both sides start from the bias and never see each other's state, so a split that
goes to another feature moves every later round.  Small nodes of integer targets hold splits of different rows whose gains
are equal in exact arithmetic; only sums without rounding noise send them to the first feature, as float64 does."""
import math

import numpy as np
import pytest

from tests.parity import _gain_of, oracle_params

pytestmark = pytest.mark.gpu

# What float64 itself can say about a gain: a sum of n terms is off by at most n 2^-53 of the sum of their magnitudes (the
# oracle adds them one by one, the library once per bin), a gain takes four such sums and a dozen operations on top.
EPS = 2.0 ** -53


def _table(n, F, seed):
    rng = np.random.default_rng(seed)
    x = rng.normal(size=(n, F)).astype(np.float32)
    x[:, 1::3] = np.exp(x[:, 1::3])
    x[:, 2::3] = np.floor(np.abs(x[:, 2::3]) * 2)
    return x, (x @ rng.normal(size=F).astype(np.float32)), rng


def _target(loss, s, rng):
    z = (s - s.mean()) / s.std()
    if loss == "poisson":
        return rng.poisson(np.exp(np.clip(0.6 * z, -4, 4))).astype(np.float32)
    if loss == "logloss":   # as many ones as zeros: the first gradients are +1/2 and -1/2
        y = (z + 0.5 * rng.normal(size=s.size)).argsort().argsort() >= s.size // 2
        return y.astype(np.float32)
    r = (z + 0.5 * rng.normal(size=s.size)).argsort().argsort()   # three classes of equal size
    return (3 * r // s.size).astype(np.int64)


def _first_difference(op, t, g, hist, nsum):
    """None, or the first node and the splits of the oracle and of the library there, with their gains by the oracle's sums."""
    ts, gs = t.split.astype(bool), g.split.astype(bool)
    for n in np.nonzero((ts != gs) | (ts & ((t.feat != g.feat) | (t.cond_bin != g.cond_bin))))[0]:
        gain = lambda tree: _gain_of(op, hist[n], nsum[n], int(tree.feat[n]) - 1, int(tree.cond_bin[n])) if tree.split[n] else op.gamma  # noqa: E731
        return [int(n) + 1] + [(bool(tree.split[n]), int(tree.feat[n]), int(tree.cond_bin[n]), gain(tree)) for tree in (t, g)]
    return None


# The last poisson table has deep trees: hundreds of nodes of a few rows.
@pytest.mark.parametrize("loss,n,F,depth,colsample,seed", [("poisson", 60_013, 77, 6, 0.7, 2), ("poisson", 60_013, 77, 6, 0.7, 3), ("poisson", 60_013, 77, 6, 0.7, 4), ("poisson", 20_011, 60, 9, 1.0, 4),
                                                           ("logloss", 40_002, 20, 7, 1.0, 5), ("mlogloss", 30_003, 28, 7, 1.0, 6)])
def test_free_running_fit_grows_the_oracles_trees(pkg, orc, loss, n, F, depth, colsample, seed):
    from evotrees_b200.fit import init_target, make_rngs
    x, s, rng = _table(n, F, seed)
    y = _target(loss, s, rng)
    cls = pkg.EvoTreeClassifier if loss == "mlogloss" else pkg.EvoTreeRegressor
    params = cls(loss=loss, nrounds=12, max_depth=depth, nbins=64, eta=0.1, colsample=colsample)
    m, cache = pkg.fit(params, x_train=x, y_train=y, return_cache=True)
    pred = cache.pred()
    cache.close()
    K, yd, _, _, _, _ = init_target(loss, y, None, params.alphas)
    op = oracle_params(orc, params, K)
    b = orc.Booster(op, orc.binarize(x, m.info["edges"]), yd, use_x_bin_T=True)
    b.pred = np.tile(m.trees[0].pred.reshape(1, -1), (n, 1)).astype(np.float32)
    js_rng, njs = make_rngs(params.seed)[1], math.ceil(colsample * F)
    for r in range(params.nrounds):
        js = np.arange(1, F + 1) if njs == F else np.sort(js_rng.choice(F, size=njs, replace=False)) + 1
        t, _, hist, nsum = b.round(None, 255, js.astype(np.uint32), want_hist=True)
        diff = _first_difference(op, t, m.trees[r + 1], hist, nsum)
        if diff is not None:
            node, want, got = diff
            # the first gradients take few values and their sums need fewer than 53 bits: exact on both sides, ties included
            assert r > 0, f"node {node} of the first tree: oracle {want}, library {got}"
            terms = abs(want[3]) + 2 * sum(nsum[node - 1][k] ** 2 / (nsum[node - 1][K + k] + op.L2) for k in range(K))
            assert abs(want[3] - got[3]) <= 8 * n * EPS * terms, f"tree {r + 1}: node {node}: oracle {want}, library {got}"
            return   # a tie within float64: either is right, and the rounds after it differ
    np.testing.assert_allclose(pred, b.pred, rtol=1e-5, atol=1e-5)
