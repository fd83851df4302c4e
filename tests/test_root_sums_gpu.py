"""Sums of the root: one number per channel whichever feature's bins it is taken from, however many bits it needs.  With rows times
bits beyond the 53 of a float64, totals over the bins of two features differ in the last place; the children's sums must not
depend on which feature's scan happens to end last."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("loss,n,F,B,tail", [("gamma", 300_007, 40, 64, 3.0), ("gaussian_mle", 300_001, 33, 32, 2.0), ("cred_var", 100_003, 20, 200, 0.5),
                                             ("gamma", 5_000_001, 24, 16, 2.0), ("mlogloss", 200_003, 12, 64, 0.0), ("mae", 70_001, 50, 64, 3.0)])
def test_children_add_up_to_the_root(pkg, loss, n, F, B, tail):
    from evotrees_b200.fit import init_target
    rng = np.random.default_rng(n)
    x = rng.integers(0, B, (n, F)).astype(np.uint8) + 1
    s = rng.normal(size=n) + x[:, F // 2] / B
    y = (np.exp(tail * s) if tail else s).astype(np.float32)
    if loss == "mlogloss":
        y = np.clip(np.floor(1.5 * s).astype(np.int64), -1, 2)
    params = {"mlogloss": pkg.EvoTreeClassifier, "gaussian_mle": pkg.EvoTreeMLE}.get(loss, pkg.EvoTreeRegressor)(loss=loss, nrounds=1, max_depth=3, nbins=B, eta=0.1)
    K, yd, ycols, mu, _, _ = init_target(loss, y, None)
    cache = pkg.init_core_binned(params, np.asfortranarray(x), yd, ycols, K, mu, None, None, None, 0, 0)
    js = np.arange(1, F + 1, dtype=np.uint32)
    try:
        for r in range(4):
            g = None if r == 0 else cache.grads().astype(np.float64)     # the gradients the next tree is grown from
            t = pkg.grow_tree(cache, params, None, js, update_grads=True)
            ns = cache.node_sums()
            assert t.split[0] == 1
            np.testing.assert_array_equal(ns[0] - ns[1], ns[2], err_msg=f"tree {r + 1}")
            if g is not None:
                for c in range(2 * K + 1):                               # exact total: rounded once, twice where both sets of sums are used
                    want = math.fsum(g[:, c])
                    assert abs(ns[0][c] - want) <= 2 * np.spacing(abs(want)), (r, c, ns[0][c], want)
    finally:
        cache.close()
