"""`m(x)` at the sizes where the choice of the inference kernel changes (one CTA per row, row groups beside staged trees, 32 rows per CTA, a
thread per row, rows wider than shared memory; `test_every_kernel` asks which one a call runs) and where chunks of rows end, against a
walk over the trees in numpy; and a packed model after its trees have changed."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _model(pkg, nfeats, depth, ntrees, K, nbins, loss, seed):
    rng = np.random.default_rng(seed)
    edges = np.sort(rng.normal(size=(nfeats, nbins - 1)), axis=1)
    trees = [pkg.Tree.bias(rng.normal(size=K).astype(np.float32))]
    for _ in range(ntrees - 1):
        t = pkg.Tree.empty(depth, K)
        nn = t.feat.size
        t.split[: nn // 2] = rng.random(nn // 2) < 0.9
        t.feat[:] = np.where(t.split, rng.integers(1, nfeats + 1, nn), 0)
        t.cond_bin[:] = np.where(t.split, rng.integers(1, nbins, nn), 0)
        t.pred[:] = 0.1 * rng.normal(size=(nn, K))
        trees.append(t)
    return pkg.EvoTree(loss, K, trees, {"edges": edges, "feattypes": np.ones(nfeats, bool)})


def _walk(m, x):
    edges = m.info["edges"].astype(x.dtype)
    xb = np.stack([1 + np.searchsorted(edges[j], x[:, j], side="left") for j in range(x.shape[1])], axis=1)
    p = np.zeros((x.shape[0], m.K), np.float32)
    leaves = np.empty((x.shape[0], len(m.trees)), np.uint32)
    r = np.arange(x.shape[0])
    for i, t in enumerate(m.trees):
        n = np.ones(x.shape[0], np.int64)
        while True:
            s = t.split[n - 1] != 0
            if not s.any():
                break
            go = xb[r, np.maximum(t.feat[n - 1] - 1, 0)] <= t.cond_bin[n - 1]
            n = np.where(s, 2 * n + (~go), n)
        leaves[:, i] = n
        p += t.pred[n - 1]
        if m.loss == "mlogloss":
            p = np.maximum(np.float32(-15), p - p.max(axis=1, keepdims=True))
    if m.loss == "mlogloss":
        p = np.exp(p)
        p /= p.sum(axis=1, keepdims=True)
    return p, leaves


@pytest.mark.parametrize("rows,nfeats,depth,ntrees,K,nbins", [
    (1, 1, 1, 1, 1, 2), (1, 10, 6, 300, 1, 32), (592, 7, 5, 20, 3, 255), (593, 7, 5, 20, 3, 255), (5_001, 130, 8, 61, 1, 64), (4_097, 30, 4, 90, 64, 33),
    (33, 1_601, 3, 9, 2, 16), (65_537, 5, 9, 12, 1, 64), (70_001, 12, 11, 5, 2, 64), (300, 60_000, 3, 3, 1, 8)])
@pytest.mark.parametrize("order,dtype", [("C", np.float32), ("F", np.float64)])
def test_predict_at_the_edges_of_the_kernel_choice(pkg, rows, nfeats, depth, ntrees, K, nbins, order, dtype):
    m = _model(pkg, nfeats, depth, ntrees, K, nbins, "mlogloss" if K > 2 else "mse", rows)
    x = np.asarray(np.random.default_rng(rows).normal(size=(rows, nfeats)), dtype=dtype, order=order)
    want, leaves = _walk(m, x)
    np.testing.assert_allclose(pkg.predict(m, x).reshape(want.shape), want, rtol=1e-5, atol=1e-6)
    assert np.array_equal(pkg.predict_leaf_idx(m, x), leaves)


ONE, MID, TILES, STAGED, WIDE = range(5)


# Trees: full ones, paths that end anywhere, one bias tree.  Rows: what a kernel takes least, a remainder of its CTAs, several chunks.
@pytest.mark.parametrize("kernel,rows,nfeats,depth,ntrees,K,nbins", [
    (ONE, 592, 9, 6, 30, 1, 64), (TILES, 593, 9, 6, 30, 1, 64), (TILES, 20_011, 28, 8, 9, 5, 64),
    (MID, 593, 5, 15, 4, 1, 64), (MID, 700, 30, 11, 3, 64, 33), (MID, 5_003, 7, 14, 6, 3, 255), (MID, 1_000, 12, 13, 5, 8, 64), (MID, 9_001, 100, 15, 3, 1, 64),
    (STAGED, 400_003, 4, 7, 12, 1, 64), (STAGED, 420_011, 3, 6, 9, 5, 255), (STAGED, 500_009, 3, 5, 5, 9, 16), (STAGED, 500_017, 2, 9, 30, 2, 33),
    (WIDE, 100, 65_000, 3, 4, 33, 8), (WIDE, 70, 40_001, 4, 5, 64, 16)])
@pytest.mark.parametrize("order,dtype", [("C", np.float32), ("F", np.float32), ("F", np.float64)])
def test_every_kernel(pkg, kernel, rows, nfeats, depth, ntrees, K, nbins, order, dtype):
    import ctypes as C
    from evotrees_b200 import _lib
    m = _model(pkg, nfeats, depth, ntrees, K, nbins, "mlogloss" if K > 2 else "mse", rows)
    for t in m.trees[1:]:                                                     # all paths of every other tree are full ones
        if depth > 2 and (t.split[0] == 0 or t is m.trees[-1]):
            nn = t.feat.size
            t.split[: nn // 2] = 1
            t.feat[: nn // 2] = np.maximum(t.feat[: nn // 2], 1)
            t.cond_bin[: nn // 2] = np.maximum(t.cond_bin[: nn // 2], 1)
    x = np.asarray(np.random.default_rng(rows).normal(size=(rows, nfeats)), dtype=dtype, order=order)
    got, ids = pkg.predict(m, x), pkg.predict_leaf_idx(m, x)
    n = (C.c_int64 * 5)()
    _lib.check(_lib.lib().evb_test_predict_plan(m._dev.handle, C.c_int32(0 if dtype == np.float32 else 2), C.c_int64(rows), C.c_int32(0), n))
    assert n[kernel] > 0, list(n)
    want, leaves = _walk(m, x)
    # float32 sums of up to 40 values of size 0.1 in the same order, a power and a division of the link behind them
    np.testing.assert_allclose(got.reshape(want.shape), want, rtol=1e-5, atol=1e-6)
    assert np.array_equal(ids, leaves)


def test_walks_end_at_the_deepest_test(pkg):
    """Arrays of depth 15 whose tests end at level 4: such a model is packed, and walked, as one of five levels; a test further down is seen
    by the next call."""
    import ctypes as C
    from evotrees_b200 import _lib
    m = _model(pkg, 9, 15, 6, 1, 64, "mse", 4)
    for t in m.trees[1:]:
        t.split[15:] = 0
        t.split[:15] = 1
        t.feat[:15], t.cond_bin[:15] = np.maximum(t.feat[:15], 1), np.maximum(t.cond_bin[:15], 1)
    x = np.random.default_rng(3).normal(size=(2_000, 9))
    n = (C.c_int64 * 5)()
    for kernel, node in ((TILES, None), (TILES, 20), (MID, 16_000)):
        if node is not None:
            while node > 0:                                                   # a path down to it
                m.trees[3].split[node], m.trees[3].feat[node], m.trees[3].cond_bin[node] = 1, 2, 30
                node = (node - 1) // 2
        want, leaves = _walk(m, x)
        np.testing.assert_allclose(pkg.predict(m, x), want[:, 0], rtol=1e-5, atol=1e-6)
        assert np.array_equal(pkg.predict_leaf_idx(m, x), leaves)
        _lib.check(_lib.lib().evb_test_predict_plan(m._dev.handle, C.c_int32(2), C.c_int64(2_000), C.c_int32(0), n))
        assert n[kernel] == 1, list(n)


@pytest.mark.parametrize("K", [1, 2, 5, 9])
@pytest.mark.parametrize("rows", [8_192, 8_193, 400_003])
def test_models_whose_paths_end_early(pkg, K, rows):
    """One deep path a tree, all others end at a few levels: lanes of launches of more than 8192 rows leave the walk where their path ends"""
    m = _model(pkg, 4, 11, 9, K, 64, "mlogloss" if K > 2 else "mse", rows + K)
    rng = np.random.default_rng(K)
    for i, t in enumerate(m.trees[1:]):
        t.split[2 ** (i % 4) - 1:] = 0
        n = 0
        while 2 * n + 2 < t.feat.size:                                        # the path of a random row, all the way down
            t.split[n], t.feat[n], t.cond_bin[n] = 1, rng.integers(1, 5), rng.integers(20, 40)
            n = 2 * n + 1 + rng.integers(2)
    x = np.random.default_rng(rows).normal(size=(rows, 4)).astype(np.float32)
    want, leaves = _walk(m, x)
    assert leaves.max() >= 2 ** 10 - 1                                        # some rows get there
    np.testing.assert_allclose(pkg.predict(m, x).reshape(want.shape), want, rtol=1e-5, atol=1e-6)
    assert np.array_equal(pkg.predict_leaf_idx(m, x), leaves)


@pytest.mark.parametrize("K", [1, 3])
def test_wide_rows_of_bins(pkg, K):
    """Rows of 7 000 bins: too wide for the kernels that keep a row in shared memory"""
    import ctypes as C
    from evotrees_b200 import _lib
    m = _model(pkg, 7_000, 6, 8, K, 16, "mlogloss" if K > 2 else "mse", K)
    x = np.random.default_rng(K).normal(size=(4_000, 7_000)).astype(np.float32)
    pkg.predict(m, x[:1])                    # the model is on the device
    n = (C.c_int64 * 5)()
    _lib.check(_lib.lib().evb_test_predict_plan(m._dev.handle, C.c_int32(-1), C.c_int64(4_000), C.c_int32(0), n))
    assert n[WIDE] > 0, list(n)
    xb = np.asfortranarray(np.stack([1 + np.searchsorted(m.info["edges"][j].astype(np.float32), x[:, j], side="left") for j in range(7_000)], axis=1).astype(np.uint8))
    np.testing.assert_allclose(pkg.predict_binned(m, xb).reshape(4_000, K), _walk(m, x)[0], rtol=1e-5, atol=1e-6)


def test_packed_model_notices_changes(pkg):
    """A tree changed in place, replaced, appended, or given another array: the next call uses the new one."""
    import copy
    m = _model(pkg, 6, 5, 8, 1, 16, "mse", 3)
    x = np.random.default_rng(0).normal(size=(100, 6))

    def check():
        for _ in range(2):
            np.testing.assert_allclose(pkg.predict(m, x), _walk(m, x)[0][:, 0], rtol=1e-5, atol=1e-6)
    check()
    m.trees[3].pred[5:, 0] += 1.0
    check()
    m.trees[2].pred = m.trees[2].pred * 2
    check()
    m.trees.append(m.trees[1])
    check()
    m.trees[4] = m.trees[5]
    check()
    m.info["edges"][2] += 0.25
    check()
    m2 = copy.deepcopy(m)
    np.testing.assert_array_equal(pkg.predict(m2, x), pkg.predict(m, x))


# Trees of more than a megabyte are packed into pinned buffers by several threads: one chunk and several, a tree per unit that
# is larger than such a buffer, small trees among large ones.
@pytest.mark.parametrize("depth,ntrees,K", [(11, 200, 1), (13, 400, 1), (9, 700, 5), (15, 3, 64)])
def test_large_models(pkg, depth, ntrees, K):
    m = _model(pkg, 9, depth, ntrees, K, 32, "mse", depth)
    m.trees[1::3] = _model(pkg, 9, 4, ntrees, K, 32, "mse", 99).trees[1::3]
    x = np.random.default_rng(1).normal(size=(50, 9))
    for _ in range(2):
        np.testing.assert_allclose(pkg.predict(m, x).reshape(50, K), _walk(m, x)[0], rtol=1e-5, atol=1e-5)
    m.trees[-1].pred[-1] += 1.0             # the last value of the last tree
    m.trees[-1].split[0], m.trees[-1].feat[0], m.trees[-1].cond_bin[0] = 1, 9, 31
    np.testing.assert_allclose(pkg.predict(m, x).reshape(50, K), _walk(m, x)[0], rtol=1e-5, atol=1e-5)


def test_trees_that_cannot_be_packed(pkg):
    """Arrays of unequal lengths, a test of a feature that does not exist: errors, not reads past the end."""
    x = np.random.default_rng(0).normal(size=(3, 6))
    for change in (lambda t: setattr(t, "cond_bin", t.cond_bin[:-1]), lambda t: setattr(t, "pred", t.pred[:4]), lambda t: t.feat.__setitem__(0, 7)):
        m = _model(pkg, 6, 5, 8, 1, 16, "mse", 3)
        m.trees[2].split[0] = 1
        change(m.trees[2])
        with pytest.raises(Exception):
            pkg.predict(m, x)


def test_work_buffers_are_bounded_in_bytes(pkg):
    """Rows of 240 KB: the buffers a call keeps are those of a 12 MB chunk (its pinned and its device side are of one size), and
    the chunks of a few rows add up to the same predictions."""
    import torch
    from evotrees_b200 import _lib
    m = _model(pkg, 60_000, 4, 5, 1, 8, "mse", 1)
    x = np.random.default_rng(2).normal(size=(1_100, 60_000)).astype(np.float32)
    want = _walk(m, x[::50])[0][:, 0]
    pkg.predict(m, x[:1])                    # the model and the context are on the device
    _lib.check(_lib.lib().evb_trim_cache(0))
    free = torch.cuda.mem_get_info(0)[0]
    got = pkg.predict(m, x)
    kept = free - torch.cuda.mem_get_info(0)[0]
    np.testing.assert_allclose(got[::50], want, rtol=1e-5, atol=1e-6)
    assert kept <= 3 * 2 * (12 << 20) + (32 << 20), kept     # three slots, binned rows beside the raw ones, granularity of the allocator


def test_kernel_time_counts_overlap_once(pkg):
    """The chunks of a call run side by side: the time during which kernels ran is no longer than the call."""
    import time
    m = _model(pkg, 16, 8, 200, 5, 64, "mlogloss", 1)
    x = np.random.default_rng(2).normal(size=(500_000, 16)).astype(np.float32)
    pkg.predict(m, x)
    for _ in range(3):
        stats = {}
        t = time.perf_counter()
        pkg.predict(m, x, stats=stats)
        assert 0.0 < stats["kernel_ms"] <= (time.perf_counter() - t) * 1e3


@pytest.mark.parametrize("K,loss", [(1, "mse"), (1, "logloss"), (2, "gaussian_mle"), (3, "mlogloss"), (5, "mlogloss"), (7, "mlogloss"), (8, "mlogloss"), (9, "mlogloss")])
@pytest.mark.parametrize("n,depth,ntrees", [(593, 5, 1), (4_737, 9, 70), (20_011, 7, 33)])
def test_incomplete_trees_row_groups_and_outputs(pkg, K, loss, n, depth, ntrees):
    """Trees whose paths end anywhere, categories, a test that every bin passes; every number of outputs that has a kernel of its own"""
    rng = np.random.default_rng(n + K)
    F, B, nn = 6, 255, 2 ** depth - 1
    edges = np.sort(rng.normal(size=(F, B - 1)).astype(np.float32), axis=1)
    ft = rng.random(F) < 0.6
    trees = []
    for _ in range(ntrees):
        split = (rng.random(nn) < 0.85) & (np.arange(nn) < nn // 2)
        for i in range(1, nn):
            split[i] &= split[(i - 1) // 2]
        feat, cond = rng.integers(0, F, nn), rng.integers(1, 256, nn)
        cond[rng.random(nn) < 0.05] = 255
        trees.append(pkg.Tree(np.where(split, feat + 1, 0).astype(np.int64), np.where(split, cond, 0).astype(np.uint8), np.zeros(nn, np.float32), np.zeros(nn, np.float32),
                              rng.normal(size=(nn, K)).astype(np.float32), split.astype(np.uint8)))
    m = pkg.EvoTree(loss, K, trees, {"edges": edges, "feattypes": ft, "feature_names": [f"f{i}" for i in range(F)], "target_levels": None, "featbins": np.full(F, B, np.uint8)})
    x = rng.normal(size=(n, F)).astype(np.float32)
    xb = np.stack([1 + np.searchsorted(edges[j], x[:, j], side="left") for j in range(F)], 1)
    p, ids = np.zeros((n, K), np.float32), np.empty((n, ntrees), np.int64)
    for t, tr in enumerate(trees):
        nid = np.ones(n, np.int64)
        for _ in range(depth - 1):
            s = tr.split[nid - 1] != 0
            f, c = np.maximum(tr.feat[nid - 1] - 1, 0), tr.cond_bin[nid - 1]
            v = xb[np.arange(n), f]
            left = np.where(ft[f], v <= c, v == c)
            nid = np.where(s, 2 * nid + ~left, nid)
        ids[:, t] = nid
        p += tr.pred[nid - 1]
        if loss == "logloss":
            p = np.clip(p, np.float32(-15), np.float32(15))
        elif loss == "gaussian_mle":
            p[:, 1] = np.maximum(np.float32(-15), p[:, 1])
        elif loss == "mlogloss":
            p = np.maximum(np.float32(-15), p - p.max(1, keepdims=True))
    assert np.array_equal(pkg.predict_leaf_idx(m, x), ids)
    got = pkg.predict(m, x).reshape(n, -1)
    p = p.astype(np.float64)
    want = {"mse": lambda: p, "logloss": lambda: 1 / (1 + np.exp(-p)), "gaussian_mle": lambda: np.stack([p[:, 0], np.log1p(np.exp(-abs(p[:, 1]))) + np.maximum(p[:, 1], 0)], 1),
            "mlogloss": lambda: np.exp(p) / np.exp(p).sum(1, keepdims=True)}[loss]()
    # the sums are the same float32 additions in the same order; the link's functions are within a few units in the last place
    np.testing.assert_allclose(got, want, rtol=2e-6, atol=1e-7)
