"""Histograms of channels whose values span many orders of magnitude: every entry has to be the float64 sum of the rows' float32
gradients, the typical row's bits included however far the largest one lies above it.  Tails from narrow (nothing is left after the
words of a row) over a few rows per piece (queue) to nearly all of them (second pass); one and several channel groups, tails of words,
255 bins, row samples of few rows per node."""
import numpy as np
import pytest

from tests.parity import oracle_params

pytestmark = pytest.mark.gpu

CASES = [  # loss, classes, rows, features, bins, depth, sigma of the log-normal target, weights, columns
    ("cred_std", 0, 60_000, 20, 64, 5, 4.0, False, 20), ("cred_var", 0, 60_001, 21, 64, 5, 4.0, False, 21), ("cred_var", 0, 3_001, 5, 255, 4, 6.0, False, 5),
    ("gamma", 0, 40_003, 33, 64, 4, 3.0, True, 20), ("poisson", 0, 70_001, 9, 32, 5, 1.2, False, 9), ("mae", 0, 50_001, 40, 64, 4, 5.0, False, 40),
    ("gaussian_mle", 0, 30_011, 50, 32, 4, 2.5, False, 50), ("gaussian_mle", 0, 2_500_009, 6, 32, 4, 1.0, False, 6), ("mse", 0, 30_000, 18, 64, 4, 6.0, True, 11),
    ("mse", 0, 20_001, 6, 200, 4, 6.0, True, 6), ("mlogloss", 4, 20_001, 12, 64, 4, 12.0, True, 12), ("logloss", 0, 400_009, 7, 64, 4, 12.0, False, 7)]


@pytest.mark.parametrize("loss,classes,n,F,B,depth,sigma,weighted,ncols", CASES)
def test_histograms_keep_small_gradients(pkg, loss, classes, n, F, B, depth, sigma, weighted, ncols):
    from evotrees_b200 import _lib
    from evotrees_b200.fit import init_target
    rng = np.random.default_rng(n + B)
    x = rng.integers(0, B, (n, F)).astype(np.uint8) + 1
    z = rng.normal(size=n)
    y, pred0 = np.exp(sigma * z).astype(np.float32), None
    if loss == "poisson":
        y = np.floor(y)
    if loss in ("logloss", "mlogloss"):   # predictions between certain and undecided: probabilities down to 1e-7 and below
        K = max(classes, 1)
        y = rng.integers(0, max(classes, 2), n)
        pred0 = np.clip(sigma / 3 * rng.normal(size=(n, K)), -15, 15).astype(np.float32)
        if K > 1:
            pred0 -= pred0.max(1, keepdims=True)
        y = y.astype(np.int64) if K > 1 else y.astype(np.float32)
    params = {"mlogloss": pkg.EvoTreeClassifier, "gaussian_mle": pkg.EvoTreeMLE}.get(loss, pkg.EvoTreeRegressor)(
        loss=loss, nrounds=1, max_depth=depth, nbins=B, eta=0.3, min_weight=1.0)
    K, yd, ycols, mu, _, _ = init_target(loss, y, None)
    w = rng.uniform(0.25, 3.0, n).astype(np.float32) if weighted else None
    cache = pkg.init_core_binned(params, np.asfortranarray(x), yd, ycols, K, mu, w, pred0, None, 0, _lib.FLAG_FULL_PARTITION | _lib.FLAG_KEEP_ALL_HIST)
    try:
        C = 2 * K + 1
        js = np.sort(rng.permutation(F)[:ncols]).astype(np.uint32) + 1
        for _ in range(3):                                            # the fourth tree is a replay of the second one's graph
            pkg.grow_tree(cache, params, None, js, update_grads=True)
        g = cache.grads().reshape(n, C).astype(np.float64)
        t = pkg.grow_tree(cache, params, None, js, update_grads=True)
        nid = cache.nidx(from_partition=True).astype(np.int64)
        level = np.floor(np.log2(nid)).astype(np.int64)
        assert t.split[0]
        root_abs = root_cnt = None
        for node in range(1, 2 ** (depth - 1)):
            if node > 1 and not t.split[node // 2 - 1]:
                continue
            d = node.bit_length() - 1
            rows = np.nonzero((level >= d) & ((nid >> np.maximum(level - d, 0)) == node))[0]
            ref = np.zeros((ncols, B, C))
            mag = np.zeros((ncols, B, C))
            for i, f in enumerate(js):
                b = x[rows, f - 1].astype(np.int64) - 1
                for c in range(C):
                    ref[i, :, c] = np.bincount(b, weights=g[rows, c], minlength=B)
                    mag[i, :, c] = np.bincount(b, weights=np.abs(g[rows, c]), minlength=B)
            if node == 1:
                root_abs, root_cnt = mag, np.stack([np.bincount(x[:, f - 1].astype(np.int64) - 1, minlength=B) for f in js])[..., None]
            h = cache.hist(node, ncols, B)
            # float64 sums of the root's rows of the cell (a sibling is a difference of them), twice: the reference's and the library's
            tol = 2 * (root_cnt + depth) * 2.0 ** -53 * root_abs + 1e-300
            assert (np.abs(h - ref) <= tol).all(), (node, (np.abs(h - ref) / tol).max((0, 1)))
    finally:
        cache.close()


@pytest.mark.parametrize("loss,weighted", [("mse", False), ("mse", True), ("poisson", False), ("gamma", False)])
def test_infinite_gradient(pkg, orc, loss, weighted):
    """One row's gradient overflows: no split has a gain then, and the only leaf is what the oracle says it is."""
    from evotrees_b200.fit import init_target
    rng = np.random.default_rng(3)
    n, F, B = 5_000, 6, 32
    x = rng.integers(0, B, (n, F)).astype(np.uint8) + 1
    y = (1 + rng.integers(0, 5, n)).astype(np.float32)
    pred0 = None
    if loss == "mse":
        y[77] = 3e38
    else:
        pred0 = np.zeros((n, 1), np.float32)
        pred0[77] = 100.0 if loss == "poisson" else -110.0
    w = rng.uniform(0.25, 3.0, n).astype(np.float32) if weighted else None
    params = pkg.EvoTreeRegressor(loss=loss, nrounds=1, max_depth=4, nbins=B)
    K, yd, ycols, mu, _, _ = init_target(loss, y, None)
    cache = pkg.init_core_binned(params, np.asfortranarray(x), yd, ycols, K, mu, w, pred0, None, 0, 0)
    try:
        js = np.arange(1, F + 1, dtype=np.uint32)
        t = pkg.grow_tree(cache, params, None, js, update_grads=True)
    finally:
        cache.close()
    op = oracle_params(orc, params, K)
    grad = np.ones((n, 3), np.float32) if w is None else np.repeat(w[:, None], 3, 1)
    orc.update_grads(op, np.tile(mu, (n, 1)).astype(np.float32) if pred0 is None else pred0, yd, grad)
    assert not np.isfinite(grad).all()
    to = orc.grow_tree(op, np.asfortranarray(x), grad, np.arange(1, n + 1, dtype=np.uint32), js)[0]
    assert not to.split.any() and not t.split.any()
    np.testing.assert_array_equal(t.pred[0], to.pred[0])
