"""The staged batch kernel's packed matrix at its edges, bit for bit against
the oracle's FP32 chain: rows short of a slice and of a pair of entries,
empty rows, rows of every length in one matrix, columns beyond the window,
the matrix resident in shared memory and streamed past it, one row per
matrix, matrices whole and in parts, more of them than thread blocks; and plans
of different windows alive together."""
import numpy as np
import pytest

import mpk_gb300 as M
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _random(n, lens, seed, spread=None):
    """Rows of the given lengths (cycled), distinct ascending columns within
    `spread` of the row (None: anywhere)."""
    rng = np.random.default_rng(seed)
    rows = []
    for i in range(n):
        lo, hi = (0, n) if spread is None else (max(0, i - spread), min(n, i + spread + 1))
        rows.append(np.sort(rng.choice(np.arange(lo, hi), size=min(lens[i % len(lens)], hi - lo), replace=False)))
    ptr = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    return M.Csr(ptr, np.concatenate(rows).astype(np.int32), rng.normal(size=int(ptr[-1])))


def _check(plan, mats, nrhs, k, seed):
    n = sum(m.n for m in mats)
    x = M.uniform(seed, n * nrhs).astype(np.float32).reshape(n, nrhs)
    vb = np.zeros((k + 1, n, nrhs), dtype=np.float32)
    want, r = [], 0
    for m in mats:
        want.append(O.spmm_f32(m.ptr, m.col, m.val.astype(np.float32), x[r:r + m.n], k))
        r += m.n
    want = np.concatenate(want, axis=1)
    for _ in range(2):  # the flags carry on from call to call
        vb[0] = x
        vb[1:] = -1
        plan.exec_batch_host(vb)
        assert vb.tobytes() == want.tobytes()


EDGES = {
    "tiny": lambda: [_random(n, [1, 2, 3], n) for n in (1, 2, 7, 31, 33)],
    "empty_rows": lambda: [_random(300, [0, 5, 0, 1, 8], 1, 40), _random(65, [0, 0, 3], 2)],
    "all_lengths": lambda: [_random(1500, list(range(70)), 3, 64)],
    "anywhere": lambda: [_random(9000, [4, 9, 1], 4), M.Csr.laplacian(30, 30, 30)],
    "whole_and_parts": lambda: [_random(n, [9, 13, 30], n, 64) for n in (300, 760, 64, 1500, 4000, 2900)],
    "more_than_ctas": lambda: [_random(1 + n % 9, [2, 3], n) for n in range(160)],
    "long_rows": lambda: [_random(700, [2, 2, 2, 600], 5), _random(257, [257], 6)],
}


@pytest.mark.parametrize("mats", EDGES)
@pytest.mark.parametrize("nrhs,k", [(4, 3), (8, 1), (16, 4), (128, 2)])
@pytest.mark.parametrize("mode", [M.BATCH_DEFAULT, M.BATCH_STAGED4])
def test_packed_rows(mats, nrhs, k, mode, gpu):
    m = EDGES[mats]()
    _check(M.Plan.batch(m, nrhs, k, tune=mode), m, nrhs, k, 3)


def test_streamed_beyond_residence(gpu):
    """A matrix larger than all the shared memory, in several groups."""
    m = [M.Csr.banded(120000, 64, 5, 30, seed=1), M.Csr.diffusion(300, 401, 1, sigma=0.5, seed=2)]
    plan = M.Plan.batch(m, 32, 2, tune=M.BATCH_STAGED2)
    assert plan.batch_info()["ngroup"] > 1
    _check(plan, m, 32, 2, 5)


def test_plans_of_different_windows(gpu):
    m = [M.Csr.banded(2000, 64, 5, 30, seed=7)]
    plans = [M.Plan.batch(m, 16, 3, tune=t) for t in (M.BATCH_STAGED, M.BATCH_STAGED4, M.BATCH_STAGED2)]
    for p in plans:
        _check(p, m, 16, 3, 9)
