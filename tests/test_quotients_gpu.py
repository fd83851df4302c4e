"""The split scan's quotients against the division of doubles."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _quotients(a, b):
    from evotrees_b200 import _lib
    a, b = np.ascontiguousarray(a, np.float64), np.ascontiguousarray(b, np.float64)
    q, ok = np.empty(a.size), np.empty(a.size, np.uint8)
    _lib.check(_lib.lib().evb_test_quotients(C.c_int32(0), C.c_int64(a.size), _lib.ptr(a), _lib.ptr(b), _lib.ptr(q), _lib.ptr(ok)))
    with np.errstate(all="ignore"):
        return q, a / b, ok.astype(bool)


def _mantissas(rng, n):
    return rng.integers(1 << 52, 1 << 53, n, dtype=np.uint64).astype(np.float64)


def test_random_pairs(pkg):
    rng = np.random.default_rng(1)
    for _ in range(8):
        n = 1 << 22
        a = np.ldexp(_mantissas(rng, n), rng.integers(-652, 547, n))         # 2^-600 .. 2^600
        b = np.ldexp(_mantissas(rng, n), rng.integers(-104, 247, n))         # 2^-52 .. 2^300
        q, want, ok = _quotients(a, b)
        assert ok.all() and np.array_equal(q, want)


def test_pairs_next_to_the_middle_of_two_numbers(pkg):
    """m b = 2^54 a +- 1 for an odd m of 54 bits: a / b is as close to m / 2^54, the middle of two doubles, as a quotient can be"""
    rng = np.random.default_rng(2)
    hard = 0
    for _ in range(8):
        m = rng.integers(1 << 53, 1 << 54, 1 << 22, dtype=np.uint64) | np.uint64(1)
        inv = m.copy()
        for _ in range(5):                                                    # Newton: the inverse modulo 2^64
            inv *= np.uint64(2) - m * inv
        inv &= np.uint64((1 << 54) - 1)
        for sign, b in ((1, inv), (-1, np.uint64(1 << 54) - inv)):
            keep = (b >= 1 << 52) & (b < 1 << 53)
            mm, bb = m[keep], b[keep]
            # a = (m b - sign) / 2^54 from halves of 27 bits; the low 54 bits of m b are sign modulo 2^54
            m1, m0, b1, b0 = mm >> np.uint64(27), mm & np.uint64((1 << 27) - 1), bb >> np.uint64(27), bb & np.uint64((1 << 27) - 1)
            mid = m1 * b0 + m0 * b1
            low = (mid & np.uint64((1 << 27) - 1)) * np.uint64(1 << 27) + m0 * b0
            a = m1 * b1 + (mid >> np.uint64(27)) + (low >> np.uint64(54)) + np.uint64(1 if sign < 0 else 0)
            a, bb = a[a >= 1 << 52], bb[a >= 1 << 52]
            hard += a.size
            q, want, ok = _quotients(a.astype(np.float64), bb.astype(np.float64))
            assert ok.all() and np.array_equal(q, want)
    assert hard > 1_000_000


def test_edges_of_the_range(pkg):
    """Zero, the ends of the range on both sides, numbers of all ones, denormals, infinities and NaN: the division either way, but for the
    last bit of the one quotient that the method is known to miss"""
    eps = np.finfo(np.float64).eps
    ones = np.nextafter(2.0, 0.0)
    a = np.array([0.0, 5e-324, 1e-310, 1e-290, 2.0 ** -601, np.nextafter(2.0 ** -600, 0), 2.0 ** -600, 1e-100, eps, 1.0, ones, 3.0, 1e100, np.nextafter(2.0 ** 600, 0), 2.0 ** 600,
                  1e290, 1e300, np.inf, np.nan])
    b = np.array([eps, np.nextafter(eps, 1), 1e-3, 0.5, ones / 2, 1.0, ones, 3.0, 1e30, np.nextafter(2.0 ** 300, 0), 2.0 ** 300, 1e290, 1e308, np.inf])
    a, b = (z.ravel() for z in np.meshgrid(a, b))
    q, want, ok = _quotients(a, b)
    # A power of two by a number of all ones: its reciprocal lies just off the middle of two numbers, Newton's iteration ends on the even one
    ties = (np.frexp(a)[0] == 0.5) & (np.frexp(b)[0] == ones / 2) & ok
    # no sum of gradients has a square between zero and 2^-600: the remainder loses bits below the smallest numbers there
    tiny = (a > 0) & (a < 2.0 ** -600) & ok
    assert np.array_equal(q[~ties & ~tiny], want[~ties & ~tiny], equal_nan=True)
    assert ties.sum() >= 9 and np.all(np.abs(q[ties | tiny] - want[ties | tiny]) <= 2 * np.spacing(want[ties | tiny]))
    assert np.array_equal(ok, (a < 2.0 ** 600) & (b < 2.0 ** 300))
    rng = np.random.default_rng(3)                                            # divisors of all ones: reciprocals next to the middle of two numbers
    a = _mantissas(rng, 1 << 20)
    q, want, ok = _quotients(a, np.ldexp(ones, rng.integers(-52, 299, a.size)))
    assert ok.all() and np.array_equal(q, want)
