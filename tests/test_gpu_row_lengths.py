"""Rows of every length around the groups that the FP64 row sums go in (8
entries ahead, then fours; fours and their remainder in the k-SpMV), in the
general wavefront and in k-SpMV launches of fewer and of more blocks than SMs,
bit for bit against the oracle."""
import numpy as np
import pytest

import mpk_gb300 as M
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _matrix(n, uniform, seed):
    """Row i has (i + i // 32) % 46 entries (slices of one length each if `uniform`), columns near it."""
    rng = np.random.default_rng(seed)
    i = np.arange(n)
    length = np.where(i // 32 % 2 == 0, i // 64 % 46, (i + i // 32) % 46) if not uniform else i // 32 % 46
    ptr = np.concatenate([[0], np.cumsum(length)]).astype(np.int32)
    row = np.repeat(i, length)
    off = np.arange(ptr[-1]) - ptr[row]
    col = np.clip(row + 3 * off - 60 - rng.integers(0, 3, n)[row], None, n - 1)
    col = np.where(col < 0, off, col).astype(np.int32)
    return M.Csr(ptr, col, rng.normal(size=int(ptr[-1])))


@pytest.mark.parametrize("plan", ["wave", "spmv"])
@pytest.mark.parametrize("n,uniform", [(3001, False), (20011, True), (60013, False)])
@pytest.mark.parametrize("valued", [False, True])
@pytest.mark.parametrize("arith", [M.ARITH_FMA, M.ARITH_SEPARATE])
def test_every_row_length(plan, n, uniform, valued, arith, gpu):
    a = _matrix(n, uniform, 3)
    a = a if valued else M.Csr(a.ptr, a.col)
    k = 3
    x = M.uniform(5, n)
    p = M.Plan.wave(a, k, arith=arith) if plan == "wave" else M.Plan.spmv(a, k, arith=arith)
    vv = np.zeros((k + 1) * n)
    vv[:n] = x
    p.exec_host(vv)
    want = O.mpk(a.ptr, a.col, a.val, x, k, O.MODE_FMA if arith == M.ARITH_FMA else O.MODE_SEPARATE)
    assert vv.tobytes() == want.tobytes()


@pytest.mark.parametrize("valued", [False, True])
@pytest.mark.parametrize("order", ["beyond_l2", "random"])
def test_rows_without_integer_products(order, valued, gpu):
    """The general wavefront where rows wait for memory: levels beyond L2, and columns anywhere."""
    if order == "random":
        a = _matrix(70001, False, 4)
        a = M.Csr(np.arange(0, 4 * a.n + 1, 4, dtype=np.int32), np.random.default_rng(1).integers(0, a.n, 4 * a.n).astype(np.int32))
    else:
        a = M.Csr.laplacian(150, 150, 151)
    a = M.Csr(a.ptr, a.col, M.uniform(3, a.nnz) if valued else None)
    k = 2
    x = M.uniform(5, a.n)
    vv = np.zeros((k + 1) * a.n)
    vv[:a.n] = x
    M.Plan.wave(a, k, ctas_per_sm=32).exec_host(vv)
    assert vv.tobytes() == O.mpk(a.ptr, a.col, a.val, x, k, O.MODE_FMA).tobytes()


@pytest.mark.parametrize("n,uniform", [(3001, False), (20011, True)])
@pytest.mark.parametrize("valued", [False, True])
@pytest.mark.parametrize("arith", [M.ARITH_FMA, M.ARITH_SEPARATE])
def test_longest_rows(n, uniform, valued, arith, gpu):
    """The general wavefront where rows have more than 28 entries on average: every length from 20 to 65."""
    i = np.arange(n)
    length = 20 + (i // 32 % 46 if uniform else i % 46)
    ptr = np.concatenate([[0], np.cumsum(length)]).astype(np.int32)
    row = np.repeat(i, length)
    first = np.clip(i - 3 * (length // 2), 0, n - 3 * 65)
    col = (first[row] + 3 * (np.arange(ptr[-1]) - ptr[row])).astype(np.int32)
    assert ptr[-1] > 28 * n
    a = M.Csr(ptr, col, np.random.default_rng(6).normal(size=int(ptr[-1])) if valued else None)
    k = 3
    x = M.uniform(5, n)
    vv = np.zeros((k + 1) * n)
    vv[:n] = x
    M.Plan.wave(a, k, arith=arith).exec_host(vv)
    want = O.mpk(a.ptr, a.col, a.val, x, k, O.MODE_FMA if arith == M.ARITH_FMA else O.MODE_SEPARATE)
    assert vv.tobytes() == want.tobytes()


@pytest.mark.parametrize("length", [65, 203, 2000])
@pytest.mark.parametrize("valued", [False, True])
@pytest.mark.parametrize("arith", [M.ARITH_FMA, M.ARITH_SEPARATE])
def test_one_long_row(length, valued, arith, gpu):
    """The general wavefront over a mesh whose level waits for one row."""
    a = M.Csr.laplacian(100, 100)
    i = 5000
    lo, hi = int(a.ptr[i]), int(a.ptr[i + 1])
    ptr = a.ptr.astype(np.int64)
    ptr[i + 1:] += length - (hi - lo)
    col = np.concatenate([a.col[:lo], i - 30 + np.arange(length), a.col[hi:]])
    a = M.Csr(ptr.astype(np.int32), col.astype(np.int32), np.random.default_rng(8).normal(size=len(col)) if valued else None)
    k = 3
    x = M.uniform(5, a.n)
    vv = np.zeros((k + 1) * a.n)
    vv[:a.n] = x
    M.Plan.wave(a, k, arith=arith, ctas_per_sm=32).exec_host(vv)
    want = O.mpk(a.ptr, a.col, a.val, x, k, O.MODE_FMA if arith == M.ARITH_FMA else O.MODE_SEPARATE)
    assert vv.tobytes() == want.tobytes()
