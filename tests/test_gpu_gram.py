"""Entries of the s-step method's Gram matrix against exact sums (math.fsum of
the products, which are exact in FP64).

An entry takes at most two additions in FP64 for each tile of 64 rows that a
block sums, one for every 32 blocks' partial sums and five across a warp, each
off by 2^-53 of the sum S of the products' magnitudes at the most; what is left
out within a tile is below 2^-58 S (64 errors' errors in FP32).  Independent
roundings of r sums have a root mean square of sqrt(r / 3) 2^-53 S.  In
double-float every sum of N values rounds N low parts of up to N 2^-24 S."""
import math

import numpy as np
import pytest

import mpk_gb300 as M

pytestmark = pytest.mark.gpu


def _exact(y):
    """Exact sums and sums of magnitudes of all the columns' products."""
    y = y.astype(np.float64)
    g, s = np.zeros((2, len(y), len(y)))
    for a in range(len(y)):
        for b in range(a, len(y)):
            p = y[a] * y[b]
            g[a, b] = g[b, a] = math.fsum(p)
            s[a, b] = s[b, a] = math.fsum(np.abs(p))
    return g, s


def _roundings(n):
    tiles = (n + 63) // 64
    blocks = min(1216, tiles)
    return 2 * -(-tiles // blocks) + -(-blocks // 32) + 5


def _normal(n, m, seed):
    rng = np.random.default_rng(seed)
    y = rng.normal(size=(m, n))
    for c in range(1, m):  # correlated, as a basis is
        y[c] = 0.7 * y[c - 1] + 0.3 * y[c]
    return y


def _sparse_range(n, m, seed):
    """Each column large on its own rows and 2^-100 elsewhere: the products of
    two columns are large nowhere, or tiny everywhere."""
    rng = np.random.default_rng(seed)
    y = (1 + rng.random((m, n))) * rng.choice([-1.0, 1.0], (m, n))
    own = np.arange(n) % (m + 3) == np.arange(m)[:, None]
    y[~own] *= 2.0 ** -100
    y[::2] *= own[::2] | (np.arange(n) % 2 == 0)  # and zeros
    return y


DATA = {
    "normal": _normal,
    "positive": lambda n, m, seed: np.abs(_normal(n, m, seed)),
    "shrinking": lambda n, m, seed: _normal(n, m, seed) * 2.0 ** (-7.0 * np.arange(m))[:, None],
    "subnormal": lambda n, m, seed: np.ldexp(_normal(n, m, seed), -140 + 3 * np.arange(m)[:, None]),
    "large": lambda n, m, seed: np.ldexp(_normal(n, m, seed), 120 - 5 * np.arange(m)[:, None]),
    "within_range": lambda n, m, seed: np.ldexp(_normal(n, m, seed), -np.random.default_rng(seed).integers(0, 36, (m, n))),
    "wide_range": lambda n, m, seed: np.ldexp(_normal(n, m, seed), -np.random.default_rng(seed).integers(0, 130, (m, n))),
    "sparse_range": _sparse_range,
    "zeros": lambda n, m, seed: _normal(n, m, seed) * (np.arange(m) % 3 > 0)[:, None],
}


@pytest.mark.parametrize("data", DATA)
@pytest.mark.parametrize("n,m", [(1, 2), (63, 3), (209, 17), (3001, 21)])
def test_entries_against_exact_sums(data, n, m, gpu):
    y = DATA[data](n, m, 7).astype(np.float32)
    want, s = _exact(y)
    err = np.abs(M.debug_gram(y) - want)
    assert np.all(err <= (_roundings(n) + 1) * 2.0 ** -53 * s)
    if n > 64:
        rel = err[s > 0] / s[s > 0]
        assert math.sqrt(np.mean(rel ** 2)) <= math.sqrt(_roundings(n) / 3) * 2.0 ** -53
    low = np.abs(M.debug_gram(y, gram=M.GRAM_DF64) - want)
    if data in ("normal", "positive", "zeros"):  # the others leave the range of its FP32 products
        terms = 16 * -(-((n + 63) // 64) // min(1216, (n + 63) // 64)) + 4
        assert np.all(low <= (terms * terms * 2.0 ** -48 + _roundings(n) * 2.0 ** -53) * s)


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
def test_infinities_and_nan(bad, gpu):
    """In their own row and column only, as FP64 gives them."""
    y = _normal(209, 9, 3).astype(np.float32)
    clean, _ = _exact(y)
    y[4, 77] = bad
    y[6, 77] = 0
    with np.errstate(invalid="ignore"):
        want = np.array([[np.sum(a.astype(np.float64) * b) for b in y] for a in y])
    got = M.debug_gram(y)
    fin = np.isfinite(want)
    assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(np.isposinf(got), np.isposinf(want))
    assert not np.isfinite(want[4]).any() and fin[:4, :4].all()
    exact, s = _exact(y[:4])
    assert np.all(np.abs(got[:4, :4] - exact) <= (_roundings(209) + 1 + 64) * 2.0 ** -53 * s)  # a tile summed in FP64
