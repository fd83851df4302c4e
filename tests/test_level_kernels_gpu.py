"""The kernels of a tree level at the edges of their tiles: histograms against float64 sums of the device's own gradients,
splits against every candidate of those histograms, row ids against the tree.  Features: every tail of the words a lane owns
(8 / 4 / 2 / 1), one and several groups; bins: 2 to 255; outputs: one, the warps of one scan CTA (2 to 8) and more; rows:
fewer than a CTA, ragged, more than one accumulation epoch of a CTA holds."""
import numpy as np
import pytest

from tests.parity import _gain_of

pytestmark = pytest.mark.gpu

CASES = [  # loss, classes, rows, features, bins, depth, weights, columns
    ("logloss", 0, 37, 1, 2, 3, False, 1), ("poisson", 0, 2_049, 7, 33, 4, False, 7), ("gamma", 0, 40_007, 33, 128, 4, True, 20),
    ("mse", 0, 30_001, 13, 255, 5, True, 13), ("mse", 0, 9_000, 21, 64, 4, False, 11), ("gaussian_mle", 0, 30_011, 9, 32, 6, False, 9),
    ("gaussian_mle", 0, 5_000, 130, 16, 4, True, 130), ("mlogloss", 3, 10_240, 15, 65, 5, False, 15), ("mlogloss", 5, 3_001, 28, 64, 5, True, 28),
    ("mlogloss", 8, 4_097, 4, 255, 5, False, 4), ("mlogloss", 9, 4_099, 5, 40, 4, False, 3), ("logloss", 0, 12_000_000, 2, 8, 3, False, 2),
    # one or two parts fit shared memory: rows cut into words of 8 and 4, tails of five words
    ("mse", 0, 90_001, 50, 255, 4, True, 50), ("logloss", 0, 90_003, 18, 255, 4, False, 18), ("poisson", 0, 90_001, 52, 128, 4, False, 52)]


@pytest.mark.parametrize("loss,classes,n,F,B,depth,weighted,ncols", CASES)
def test_level_kernels(pkg, loss, classes, n, F, B, depth, weighted, ncols):
    from evotrees_b200 import _lib
    from evotrees_b200.fit import init_target
    rng = np.random.default_rng(n + F)
    x = rng.integers(0, B, (n, F)).astype(np.uint8) + 1
    s = x[:, 0].astype(np.float32) / B + 0.5 * rng.random(n, dtype=np.float32) + (x[:, F // 2] > B // 2)
    y = {"logloss": lambda: (s > 1).astype(np.float32), "poisson": lambda: np.floor(3 * s), "gamma": lambda: s + 0.1,
         "mlogloss": lambda: np.minimum((s * classes / 2.6).astype(np.int64), classes - 1)}.get(loss, lambda: s)()
    if loss == "mlogloss":
        y[:classes] = np.arange(classes)
    params = {"mlogloss": pkg.EvoTreeClassifier, "gaussian_mle": pkg.EvoTreeMLE}.get(loss, pkg.EvoTreeRegressor)(
        loss=loss, nrounds=1, max_depth=depth, nbins=B, eta=0.3, min_weight=1.0, **({"lambda_": 0.1} if n % 2 else {}))
    K, yd, ycols, mu, _, _ = init_target(loss, y, None)
    w = rng.uniform(0.25, 3.0, n).astype(np.float32) if weighted else None
    cache = pkg.init_core_binned(params, np.asfortranarray(x), yd, ycols, K, mu, w, None, None, 0,
                                 _lib.FLAG_FULL_PARTITION | _lib.FLAG_KEEP_ALL_HIST)
    try:
        C = 2 * K + 1
        allf = np.arange(1, F + 1, dtype=np.uint32)
        pkg.grow_tree(cache, params, None, allf, update_grads=True)   # leaves the gradients of the next round
        g = cache.grads().reshape(n, C).astype(np.float64)
        js = np.sort(rng.permutation(F)[:ncols]).astype(np.uint32) + 1
        t = pkg.grow_tree(cache, params, None, js, update_grads=True)
        nid = cache.nidx(from_partition=True).astype(np.int64)
        op = type("P", (), dict(loss=loss, lambda_=params.lambda_, L2=params.L2))
        level = np.floor(np.log2(nid)).astype(np.int64)
        assert t.split[0]
        for node in range(1, 2 ** (depth - 1)):
            if node > 1 and not t.split[node // 2 - 1]:
                continue
            d = node.bit_length() - 1
            rows = np.nonzero((level >= d) & ((nid >> np.maximum(level - d, 0)) == node))[0]
            ref = np.zeros((ncols, B, C))
            for i, f in enumerate(js):
                b = x[rows, f - 1].astype(np.int64) - 1
                for c in range(C):
                    ref[i, :, c] = np.bincount(b, weights=g[rows, c], minlength=B)
            h = cache.hist(node, ncols, B)
            tol = np.maximum(np.abs(g).max(0), 1e-30) * max(rows.size, 1) * (2.0 ** -23 if loss == "mse" else 2.0 ** -28)
            assert (np.abs(h - ref) <= tol).all(), (node, np.abs(h - ref).max((0, 1)) / tol)
            tot = ref[0].sum(0)
            # every candidate's gain from the reference histogram
            left = np.cumsum(ref, axis=1)[:, :-1]
            right = tot - left

            def term(s):
                return (s[..., :K] ** 2 / np.maximum(2.2e-16, s[..., K:2 * K] + (params.lambda_ * s[..., -1] + params.L2)[..., None]) / 2).sum(-1)
            gains = term(left) + term(right) - term(tot)
            gains[(left[..., -1] <= params.min_weight) | (right[..., -1] <= params.min_weight)] = -np.inf
            best, scale = gains.max(initial=-np.inf), term(tot) + np.abs(gains[np.isfinite(gains)]).max(initial=0.0)
            if t.split[node - 1]:
                i = int(np.nonzero(js == t.feat[node - 1])[0][0])
                mine = _gain_of(op, ref, tot, i, int(t.cond_bin[node - 1]))
                assert mine >= best - 1e-5 * scale and abs(t.gain[node - 1] - mine) <= 1e-5 * scale, (node, mine, best)
                go = x[rows, t.feat[node - 1] - 1] <= t.cond_bin[node - 1]
                child = nid[rows] >> np.maximum(level[rows] - d - 1, 0)
                assert np.array_equal(child == 2 * node, go), node
            else:
                assert best <= params.gamma + 1e-5 * scale, (node, best)
    finally:
        cache.close()


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("n", [5_000, 320_000])
def test_hessians_of_least_squares_can_be_accumulated(pkg, orc, monkeypatch, weighted, n):
    """EVB_NO_ELISION: the hessian channel of mse is summed like any other instead of rebuilt from the weights."""
    from tests.parity import lockstep_check
    monkeypatch.setenv("EVB_NO_ELISION", "1")
    rng = np.random.default_rng(n)
    x = rng.random((n, 9)).astype(np.float32)
    y = (x @ rng.normal(size=9) + 0.1 * rng.normal(size=n)).astype(np.float32)
    w = rng.uniform(0.25, 3.0, n).astype(np.float32) if weighted else None
    lockstep_check(pkg, orc, pkg.EvoTreeRegressor(loss="mse", nrounds=2, max_depth=5, nbins=32, eta=0.3), x, y, rounds=2, w=w)
