"""The diagonal wavefront in each of its modes, by name: that a plan runs it,
how many levels per exchange it takes (whole blocks of them and a short last
one), and rows off the diagonals; bit for bit the general wavefront's results
(mixed forms: the FP32 oracle's).  Plans of it on two streams at once."""
import numpy as np
import pytest

import mpk_gb300 as M
from oracle import oracle as O

pytestmark = pytest.mark.gpu

ALL, PAIR, DEEP = range(3)


def _scattered(a, every, near, seed):
    """One row of every `every`-th slice with 7 columns within `near` (None: anywhere)."""
    rng = np.random.default_rng(seed)
    cols = [a.col[a.ptr[i]:a.ptr[i + 1]] for i in range(a.n)]
    for i in range(5, a.n, 32 * every):
        c = rng.integers(0, a.n, 7) if near is None else np.clip(i + rng.integers(-near, near, 7), 0, a.n - 1)
        cols[i] = np.unique(c).astype(np.int32)
    ptr = np.concatenate([[0], np.cumsum([len(c) for c in cols])]).astype(np.int32)
    return M.Csr(ptr, np.concatenate(cols).astype(np.int32), rng.normal(size=int(ptr[-1])))


CASES = {  # matrix, levels, mode, rows off the diagonals
    "all": (lambda: M.Csr.diffusion(1000, 1001, 1, sigma=0.5, seed=1), 3, ALL, False),
    "pair": (lambda: M.Csr.laplacian(90, 80, 70), 3, PAIR, False),
    "deep": (lambda: M.Csr.laplacian(100, 100), 8, DEEP, False),
    "deep_short_last": (lambda: M.Csr.laplacian(120, 110), 11, DEEP, False),
    "all_irregular": (lambda: _scattered(M.Csr.laplacian(700, 701), 25, 4000, 3), 3, ALL, True),
    "pair_irregular": (lambda: _scattered(M.Csr.laplacian(90, 80, 70), 25, 4000, 4), 3, PAIR, True),
    "pair_irregular_anywhere": (lambda: _scattered(M.Csr.laplacian(90, 80, 70), 60, None, 5), 3, PAIR, True),
}


def _is(plan, k, mode, irregular):
    got = plan.debug_diag()
    assert got is not None and got[0] == mode, got
    assert (got[1] > 1) == (mode == DEEP) and (got[2] > 0) == irregular, got
    return got[1]


@pytest.mark.parametrize("name", CASES)
@pytest.mark.parametrize("valued", [False, True])
@pytest.mark.parametrize("arith", [M.ARITH_FMA, M.ARITH_SEPARATE, M.ARITH_DF64])
def test_modes(name, valued, arith, gpu):
    make, k, mode, irregular = CASES[name]
    a = make()
    a = M.Csr(a.ptr, a.col, M.uniform(3, a.nnz) if valued else None)
    x = M.uniform(5, a.n)
    got, want = np.zeros((2, (k + 1) * a.n))
    got[:a.n] = want[:a.n] = x
    plan = M.Plan.wave(a, k, arith=arith)
    depth = _is(plan, k, mode, irregular)
    assert name != "deep_short_last" or k % depth
    plan.exec_host(got)
    other = M.Plan.wave(a, k, arith=arith, ctas_per_sm=32)
    assert other.debug_diag() is None
    other.exec_host(want)
    assert got.tobytes() == want.tobytes()


@pytest.mark.parametrize("name", [c for c in CASES if not c.endswith("anywhere")])  # which mixed plans refuse
@pytest.mark.parametrize("vt", [M.VALUE_F32, M.VALUE_BF16])
def test_mixed_modes(name, vt, gpu):
    import torch
    make, k, mode, irregular = CASES[name]
    a = make()
    val = M.uniform(7, a.nnz)
    if vt == M.VALUE_BF16:
        val = (val.astype(np.float32).view(np.uint32) & 0xFFFF0000).view(np.float32).astype(np.float64)
    a = M.Csr(a.ptr, a.col, val)
    plan = M.Plan.mixed(a, k, vt)
    _is(plan, k, mode, irregular)
    e, _ = plan.mixed_scale()
    x = M.uniform(9, a.n).astype(np.float32)
    d = torch.zeros((k + 1) * a.n, dtype=torch.float32, device="cuda")
    d[:a.n] = torch.from_numpy(x).cuda()
    torch.cuda.synchronize()
    plan.exec_mixed_device(d.data_ptr())
    plan.sync()
    want = O.spmm_f32(a.ptr, a.col, (a.val * 2.0 ** -e).astype(np.float32), x[:, None], k)[:, :, 0]
    assert d.cpu().numpy().reshape(k + 1, a.n).tobytes() == want.tobytes()


def test_plans_on_two_streams(gpu):
    import torch
    k = 6
    mats = [M.Csr.laplacian(100, 100), M.Csr.diffusion(90, 91, 1, sigma=0.5, seed=2)]
    plans = [M.Plan.wave(a, k) for a in mats]
    streams = [torch.cuda.Stream() for _ in mats]
    d = [torch.zeros(((k + 1) * a.n), dtype=torch.float64, device="cuda") for a in mats]
    x = [M.uniform(q, a.n) for q, a in enumerate(mats)]
    for q, a in enumerate(mats):
        d[q][:a.n] = torch.from_numpy(x[q]).cuda()
    torch.cuda.synchronize()
    for _ in range(50):
        for p, s, v in zip(plans, streams, d):
            p.exec_device(v.data_ptr(), s.cuda_stream)
    for p, s in zip(plans, streams):
        p.sync(s.cuda_stream)
    for q, a in enumerate(mats):
        assert d[q].cpu().numpy().tobytes() == O.mpk(a.ptr, a.col, a.val, x[q], k, O.MODE_FMA).tobytes()
