"""Trees grown in one launch against the kernels of single levels on the same data: the same integers are summed, so trees, leaves,
predictions, node sums and histograms are equal bit for bit.  Rows: fewer than a tile, ragged ranges, one range and many; features: every
remainder of a word, one group and many; bins: each number a lane scans, 2 to 255; every record layout."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _data(n, F, B, loss, seed, weighted):
    rng = np.random.default_rng(seed)
    x = np.asfortranarray(rng.integers(0, B, (n, F)).astype(np.uint8) + 1)
    s = x[:, 0].astype(np.float32) / B + (x[:, F // 2] > B // 2) + 0.5 * rng.random(n, dtype=np.float32)
    y = {"logloss": lambda: (s > 1).astype(np.float32), "poisson": lambda: np.floor(3 * s), "gamma": lambda: s + 0.1,
         "tweedie": lambda: np.maximum(s - 0.6, 0)}.get(loss, lambda: s)().astype(np.float32)
    return x, y, rng.uniform(0.25, 3.0, n).astype(np.float32) if weighted else None


def _cache(pkg, params, x, y, w, flags, feattypes=None, pred0=None):
    from evotrees_b200.fit import init_target
    K, yd, ycols, mu, _, _ = init_target(params.loss, y, None)
    return pkg.init_core_binned(params, x, yd, ycols, K, mu, w, pred0, feattypes, 0, flags)


def _same(pkg, params, x, y, w, rounds=3, feattypes=None, pred0=None, grows=True, samples=None):
    """`rounds` trees of both; the handle that partitions the last level too runs the level kernels"""
    from evotrees_b200 import _lib
    keep = _lib.FLAG_KEEP_ALL_HIST
    a, b = (_cache(pkg, params, x, y, w, flags, feattypes, pred0) for flags in (keep, keep | _lib.FLAG_FULL_PARTITION))
    F = x.shape[1]
    try:
        for r in range(rounds):
            mask, js = samples[r % len(samples)] if samples else (None, np.arange(1, F + 1, dtype=np.uint32))
            s, t = (pkg.grow_tree(c, params, mask, js, update_grads=True) for c in (a, b))
            for k in ("feat", "cond_bin", "split", "w", "gain", "pred"):
                assert np.array_equal(getattr(s, k), getattr(t, k), equal_nan=k in ("w", "gain", "pred")), (r, k)
            assert np.array_equal(a.nidx(), b.nidx()) and np.array_equal(a.pred(), b.pred(), equal_nan=True)
            assert np.array_equal(a.grads(), b.grads(), equal_nan=True)
            ns, nt = a.node_sums(), b.node_sums()
            assert np.array_equal(ns, nt, equal_nan=True)
            for node in range(1, 2 ** (params.max_depth - 1)):
                if node == 1 or s.split[node // 2 - 1]:
                    assert np.array_equal(a.hist(node, js.size, params.nbins), b.hist(node, js.size, params.nbins), equal_nan=True), node
        assert (a.timings()["launches"]["scan"] == 0) == grows and b.timings()["launches"]["scan"] > 0
    finally:
        a.close(), b.close()
    return s


CASES = [  # loss, rows, features, bins, depth, weights
    ("mse", 1, 1, 2, 2, False), ("logloss", 31, 3, 16, 3, False), ("mse", 33, 4, 32, 3, True), ("poisson", 4_096, 5, 33, 4, False),
    ("poisson", 4_097, 7, 64, 5, True), ("gamma", 9_999, 8, 65, 5, False), ("tweedie", 20_011, 33, 128, 6, False), ("mse", 12_345, 13, 129, 5, False),
    ("logloss", 3_001, 6, 255, 4, True), ("mse", 100_003, 10, 32, 6, False), ("mse", 50_021, 100, 64, 5, False), ("logloss", 299_999, 28, 64, 5, False),
    ("mse", 70_001, 61, 64, 6, True), ("poisson", 2_000, 130, 64, 4, False), ("mse", 290_000, 3, 33, 9, False), ("logloss", 40_000, 4, 16, 9, False), ("mse", 40_000, 4, 16, 10, False),
    # small nodes: rows straight to the sums, images of fewer columns
    ("poisson", 5_031, 5, 64, 7, False), ("logloss", 6_443, 79, 128, 7, True), ("mse", 11_639, 30, 255, 8, False), ("gamma", 16_577, 22, 64, 8, True),
    ("mse", 2_245, 9, 128, 6, False), ("tweedie", 63_211, 11, 255, 6, False), ("mse", 190_000, 33, 64, 7, True), ("poisson", 353_000, 11, 64, 7, False)]


@pytest.mark.parametrize("loss,n,F,B,depth,weighted", CASES)
def test_same_trees(pkg, loss, n, F, B, depth, weighted):
    params = pkg.EvoTreeRegressor(loss=loss, nrounds=1, max_depth=depth, nbins=B, eta=0.3, min_weight=1.0)
    _same(pkg, params, *_data(n, F, B, loss, n + F, weighted))


@pytest.mark.parametrize("loss,weighted", [("mse", False), ("mse", True), ("logloss", False), ("gamma", True)])
def test_samples_of_rows_and_columns(pkg, loss, weighted):
    """Row masks, column samples that differ from tree to tree in number, trees that use neither in between"""
    n, F, rng = 15_013, 23, np.random.default_rng(5)
    x, y, w = _data(n, F, 64, loss, 3, weighted)
    js = [np.arange(1, F + 1, dtype=np.uint32)] + [np.sort(rng.permutation(F)[:k]).astype(np.uint32) + 1 for k in (9, 1)]
    mask = rng.integers(0, 256, n, dtype=np.uint8)
    params = pkg.EvoTreeRegressor(loss=loss, nrounds=1, max_depth=6, nbins=64, eta=0.3, rowsample=0.4)
    _same(pkg, params, x, y, w, rounds=8, samples=[(m, j) for j in js for m in (mask, None)])


# rows, columns, depth, loss, weights, numbers of sampled columns of the trees one after the other
COLUMN_COUNTS = [(2_000, 400, 5, "mse", False, (400, 200, 400, 100)), (5_000, 300, 5, "mse", True, (300, 100, 300, 150)), (2_500, 64, 5, "tweedie", True, (64, 32, 64, 16)),
                 (900, 100, 5, "logloss", True, (100, 30, 100, 7)), (1_100, 60, 4, "poisson", True, (60, 20, 60, 5, 33)), (900, 33, 6, "gamma", False, (33, 4, 30, 9))]


@pytest.mark.parametrize("n,F,depth,loss,weighted,counts", COLUMN_COUNTS)
def test_another_number_of_columns_in_every_tree(pkg, n, F, depth, loss, weighted, counts):
    """One range of rows stores its sums, several add theirs up: what a tree leaves behind must not be found by the next, whose geometry is another.
    Every tree is that of a handle which starts from the same predictions.  Gradients over many orders of magnitude, so that the second set of sums
    is used too (the level kernels round such sums elsewhere: they are compared where all fit a double)."""
    from evotrees_b200 import _lib
    x, y, w = _data(n, F, 64, loss, 11, weighted)
    rng = np.random.default_rng(n)
    js = [(np.sort(rng.permutation(F)[:k]) + 1).astype(np.uint32) for k in counts]
    params = pkg.EvoTreeRegressor(loss=loss, nrounds=1, max_depth=depth, nbins=64, eta=0.3)
    _same(pkg, params, x, y, None, rounds=2 * len(js), samples=[(None, j) for j in js])
    if loss == "gamma" and w is None:
        y = np.exp(4.0 * rng.normal(size=n)).astype(np.float32)
    elif w is not None:
        w = np.exp(4.0 * rng.normal(size=n)).astype(np.float32)
    a = _cache(pkg, params, x, y, w, _lib.FLAG_KEEP_ALL_HIST)
    try:
        for r in range(2 * len(js)):
            j = js[r % len(js)]
            b = _cache(pkg, params, x, y, w, _lib.FLAG_KEEP_ALL_HIST, pred0=a.pred())
            s, t = (pkg.grow_tree(c, params, None, j, update_grads=True) for c in (a, b))
            same = [np.array_equal(getattr(s, k), getattr(t, k)) for k in ("feat", "cond_bin", "split", "w", "gain", "pred")] + [np.array_equal(a.node_sums(), b.node_sums())]
            same += [np.array_equal(a.hist(node, j.size, 64), b.hist(node, j.size, 64)) for node in range(1, 2 ** (depth - 1)) if node == 1 or s.split[node // 2 - 1]]
            b.close()
            assert all(same) and np.isfinite(s.pred).all(), (r, same)
        assert a.timings()["launches"]["scan"] == 0
    finally:
        a.close()


def test_categories_and_constraints(pkg):
    n, F = 30_011, 9
    x, y, w = _data(n, F, 40, "logloss", 8, False)
    params = pkg.EvoTreeRegressor(loss="logloss", nrounds=1, max_depth=6, nbins=40, eta=0.3, monotone_constraints={1: 1, 5: -1})
    t = _same(pkg, params, x, y, w, feattypes=np.array([1, 0, 1, 0, 0, 1, 1, 1, 0], bool))
    assert (t.split != 0).sum() > 5


@pytest.mark.parametrize("n,depth", [(3_000, 5), (3_000, 7), (60_000, 5), (30_000, 8)])
@pytest.mark.parametrize("loss", ["gamma", "mse"])
def test_wide_ranges(pkg, loss, n, depth):
    """Gradients over many orders of magnitude: the second set of sums; infinities of one sign and of both"""
    x, y, w = _data(n, 6, 64, loss, 4, loss == "mse")
    params = pkg.EvoTreeRegressor(loss=loss, nrounds=1, max_depth=depth, nbins=64, eta=0.3)
    rng = np.random.default_rng(n)
    wide = np.exp(5.0 * rng.normal(size=n)).astype(np.float32)
    _same(pkg, params, x, wide, w, rounds=2)
    few = y.copy()
    few[:: n // 40] *= np.float32(2.0 ** 30)
    _same(pkg, params, x, few, w, rounds=2)
    if loss == "mse":   # gradients 2 (p - y) w
        for signs in (1.0, np.where(np.arange(n) % 2, 1.0, -1.0)):
            far = np.where(np.arange(n) % 100 == 7, 3e38 * signs, 0.0).astype(np.float32)
            _same(pkg, params, x, y, w, rounds=1, pred0=far[:, None])


def test_deeper_than_the_rows_carry(pkg):
    """Nodes that stop at every level, leaves of all depths, trees without a split"""
    x, y, _ = _data(2_500, 11, 32, "mse", 6, False)
    for gamma, mw in ((0.0, 1.0), (3.0, 60.0), (1e9, 1.0)):
        _same(pkg, pkg.EvoTreeRegressor(loss="mse", nrounds=1, max_depth=8, nbins=32, eta=0.3, gamma=gamma, min_weight=mw), x, y, None)


# 16 CTAs to 49 152 rows, 148 to 454 656: inside the tree's launch; more of them in launches of their own
@pytest.mark.parametrize("n,ev,F,own", [(1_503, 501, 7, False), (30_000, 40_003, 40, False), (5_000, 1, 3, False), (1_503, 49_153, 7, True), (1_503, 300_007, 7, True), (20_000, 460_001, 6, True)])
def test_metric_of_every_tree(pkg, orc, n, ev, F, own):
    """Evaluation rows in the tree's launch or behind it: the metric of each tree is that of the model's own predictions"""
    rng = np.random.default_rng(n)
    x, xe = rng.random((n, F)).astype(np.float32), rng.random((ev, F)).astype(np.float32)
    beta = rng.normal(size=F)
    y, ye = ((z @ beta + 0.1 * rng.normal(size=len(z))).astype(np.float32) for z in (x, xe))
    we = rng.uniform(0.5, 2.0, ev).astype(np.float32)
    m, cache = pkg.fit(pkg.EvoTreeRegressor(loss="mse", nrounds=12, max_depth=5, nbins=32, eta=0.3, bagging_size=1, early_stopping_rounds=100), x_train=x, y_train=y, x_eval=xe,
                       y_eval=ye, w_eval=we, return_cache=True)
    launches = cache.timings()["launches"]
    assert launches["scan"] == 0 and (launches["finalize"] >= 12) == own
    np.testing.assert_allclose(cache.pred(), m(x).reshape(n, 1), rtol=1e-5, atol=1e-6)
    cache.close()
    for i in (0, 1, 5, 12):
        p = m(xe, ntree_limit=i + 1).reshape(-1).astype(np.float64)
        # float32 predictions, float32 squares of each row: 2^-23 of a square each
        np.testing.assert_allclose(m.info["logger"]["metrics"][i], np.average((p - ye) ** 2, weights=we), rtol=2e-5)


def test_bags_and_replays(pkg):
    """Bags share their gradients; many trees one after the other leave no sums behind"""
    x, y, w = _data(20_003, 12, 64, "poisson", 9, False)
    from evotrees_b200 import _lib
    params = pkg.EvoTreeRegressor(loss="poisson", nrounds=7, max_depth=6, nbins=64, eta=0.3, bagging_size=3, colsample=0.6)
    out = []
    for flags in (0, _lib.FLAG_FULL_PARTITION):
        c = _cache(pkg, params, x, y, w, flags)
        m = pkg.EvoTree("poisson", 1, [], {"nrounds": 0})
        pkg.grow_rounds(m, c, params, 7)
        out.append((np.concatenate([t.pred for t in m.trees]), c.pred()))
        c.close()
    assert len(m.trees) == 21 and all(np.array_equal(p, q) for p, q in zip(*out))


def test_handles_side_by_side(pkg):
    """Handles of several threads on streams of their own: whole-GPU launches, clusters, level kernels and inference at the same time"""
    from concurrent.futures import ThreadPoolExecutor
    shapes = [("mse", 100_003, 10, 32, 6), ("logloss", 1_503, 7, 64, 5), ("poisson", 60_013, 40, 64, 6), ("mse", 300_007, 40, 64, 6), ("gamma", 3_001, 9, 64, 7), ("mse", 100_003, 10, 32, 6)]

    def run(s):
        loss, n, F, B, depth = s
        x, y, w = _data(n, F, B, loss, n + F, False)
        params = pkg.EvoTreeRegressor(loss=loss, nrounds=1, max_depth=depth, nbins=B, eta=0.2)
        c = _cache(pkg, params, x, y, w, 0)
        try:
            m = pkg.EvoTree(loss, 1, [], {"edges": np.sort(np.random.default_rng(F).random((F, B - 1)).astype(np.float32), axis=1), "feattypes": np.ones(F, bool), "nrounds": 0})
            out = []
            for _ in range(4):
                pkg.grow_rounds(m, c, params, 10)
                out.append(pkg.predict(m, (x[:5_000] / B).astype(np.float32)))
            return np.concatenate([t.pred for t in m.trees]), c.pred(), np.stack(out)
        finally:
            c.close()

    alone = [run(s) for s in shapes]
    with ThreadPoolExecutor(len(shapes)) as pool:
        for a, b in zip(alone, pool.map(run, shapes)):
            assert all(np.array_equal(p, q) for p, q in zip(a, b))
