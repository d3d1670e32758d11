"""FP64 rows whose products run on the integer pipes, bit for bit against the
oracle in both arithmetic modes: zeros of both signs, subnormals, values and
matrix entries whose products leave the integer range on either side or
overflow, infinities, powers of two, ties, and rows of 0 to 20 entries."""
import numpy as np
import pytest

import mpk_gb300 as M
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _values(rng, n, kind):
    v = rng.normal(size=n)
    if kind == "wide":  # exponents over the whole range
        v = np.ldexp(1.0 + rng.random(n), rng.integers(-1070, 1000, n)) * rng.choice([-1.0, 1.0], n)
    elif kind == "few_bits":  # short significands: exact products and ties
        v = rng.integers(-2**27, 2**27, n) * np.ldexp(1.0, rng.integers(-30, 30, n))
    elif kind == "special":
        v[rng.random(n) < 0.5] = 1.0
        for s in (0.0, -0.0, 5e-324, -2.3e-308, 1e308, np.inf, -np.inf, 2.0**-504, 2.0**-503, 2.0**496, 2.0**497,
                  np.nextafter(1.0, 2.0), np.nextafter(2.0, 1.0)):
            v[rng.integers(0, n, max(1, n // 60))] = s
    return v


@pytest.mark.parametrize("kind", ["normal", "wide", "few_bits", "special"])
@pytest.mark.parametrize("make", [M.Plan.wave, M.Plan.spmv])
@pytest.mark.parametrize("valued", [True, False])
def test_products_bitwise(kind, make, valued, gpu):
    rng = np.random.default_rng(5)
    n, k = 3001, 2
    rows = [np.sort(rng.choice(n, size=i % 21, replace=False)) if i % 3 else
            np.unique(np.clip(i + np.arange(-4, 5), 0, n - 1)) for i in range(n)]
    ptr = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    col = np.concatenate(rows).astype(np.int32)
    a = M.Csr(ptr, col, _values(rng, len(col), kind) if valued else None)
    x = _values(rng, n, kind)
    for arith, mode in ((M.ARITH_FMA, O.MODE_FMA), (M.ARITH_SEPARATE, O.MODE_SEPARATE)):
        with np.errstate(all="ignore"):
            want = O.mpk(a.ptr, a.col, a.val, x, k, mode)
        vv = np.zeros((k + 1) * n)
        vv[:n] = x
        plan = make(a, k, arith=arith)
        plan.exec_host(vv)
        plan.close()
        nan = np.isnan(want)
        assert np.array_equal(np.isnan(vv), nan)
        assert vv[~nan].tobytes() == want[~nan].tobytes()
