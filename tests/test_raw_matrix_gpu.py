"""Edges and bins that the device takes from a raw matrix against the host's: the sample's quantiles for every element
type and memory order, samples of one row to more rows than a CTA has threads, ties, infinities; bins in the training layouts."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,f,nbins", [(1, 3, 8), (2, 1, 2), (37, 5, 3), (1_025, 17, 64), (70_001, 20, 64), (300_000, 3, 255), (9_999, 130, 2)])
@pytest.mark.parametrize("dtype,order", [(np.float32, "C"), (np.float32, "F"), (np.float64, "C"), (np.float64, "F")])
def test_edges_equal_the_hosts(pkg, n, f, nbins, dtype, order):
    from evotrees_b200.binning import RawMatrix, sample_rows
    rng = np.random.default_rng(n + f)
    x = rng.normal(size=(n, f))
    x[:, 1::3] = np.floor(np.abs(x[:, 1::3]) * 2) * rng.choice([-1, 1], size=x[:, 1::3].shape)   # ties, both zeros
    x[:, 2::5] = np.exp(8 * x[:, 2::5])
    x = np.asarray(x, dtype=dtype, order=order)
    if n > 100:
        x[:3, 0], x[3:5, 0] = np.inf, -np.inf
    want = pkg.get_edges(x, nbins, np.random.default_rng(9))[0]
    with RawMatrix(x) as m:
        got = m.edges(nbins, sample_rows(n, nbins, np.random.default_rng(9)))
    assert got.dtype == want.dtype
    np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("n,f", [(1, 1), (257, 16), (1_000, 19), (513, 35), (300, 150)])
@pytest.mark.parametrize("order", ["C", "F"])
def test_handle_from_matrix_equals_handle_from_bins(pkg, n, f, order):
    """Same tree and training predictions as from the binned matrix: the bins reached every layout."""
    from evotrees_b200.binning import RawMatrix
    from evotrees_b200.fit import init_core_binned, init_target
    rng = np.random.default_rng(f)
    x = np.asarray(rng.normal(size=(n, f)), dtype=np.float32, order=order)
    for loss, y in (("mse", x.sum(axis=1) + x[:, -1] ** 2), ("logloss", (x[:, -1] > 0).astype(np.float32))):
        params = pkg.EvoTreeRegressor(loss=loss, nrounds=1, max_depth=4, nbins=32, min_weight=0.0)
        edges = pkg.get_edges(x, 32, np.random.default_rng(1))[0]
        K, yd, ycols, mu, _, _ = init_target(loss, y, None)
        if loss == "logloss":
            mu[:] = 0.1
        with RawMatrix(x) as m:
            a = init_core_binned(params, None, yd, ycols, K, mu, edges=edges, matrix=m)
        b = init_core_binned(params, pkg.binarize(x, edges), yd, ycols, K, mu)
        js = np.arange(1, f + 1, dtype=np.uint32)
        for _ in range(2):
            ta, tb = (pkg.grow_tree(c, params, None, js, True) for c in (a, b))
            for k in ("feat", "cond_bin", "split", "w", "gain", "pred"):
                assert np.array_equal(getattr(ta, k), getattr(tb, k)), k
        assert np.array_equal(a.pred(), b.pred())
        a.close()
        b.close()


@pytest.mark.parametrize("n", [5, 2_047, 2_052, 40_003])
def test_masks_made_on_the_device_are_the_generators(pkg, n):
    """Trees whose row masks come from the device equal trees that are given the masks, and the generator ends in the same
    place; row counts that leave half an output over included."""
    rng = np.random.default_rng(n)
    x = rng.random((n, 6)).astype(np.float32)
    y = x.sum(axis=1).astype(np.float32)
    params = pkg.EvoTreeRegressor(nrounds=5, max_depth=3, nbins=16, rowsample=0.6, min_weight=0.0)
    ma, a = pkg.init_core(params, x, y)
    mb, b = pkg.init_core(params, x, y)
    pkg.grow_rounds(ma, a, params, 3)
    pkg.grow_evotree(ma, a, params)
    for _ in range(4):
        mask, js = pkg.sample_round(b, params)
        mb.trees.append(pkg.grow_tree(b, params, mask, js, True))
    for ta, tb in zip(ma.trees, mb.trees):
        assert all(np.array_equal(getattr(ta, k), getattr(tb, k)) for k in ("feat", "cond_bin", "w", "pred"))
    assert np.array_equal(a.pred(), b.pred())
    assert np.array_equal(a.rng.integers(0, 256, 9, dtype=np.uint8), b.rng.integers(0, 256, 9, dtype=np.uint8))
    a.close()
    b.close()
