"""The diagonal wavefront (matrices whose rows keep to 5, 7 or 9 diagonals)
against the general wavefront (the same plan with a cap on its CTAs per SM)
bit for bit in FP64 and double-float, and against the oracle's FP32 chain in
the mixed form: meshes whose far diagonals lie inside and outside a CTA's own
rows, several levels per exchange of neighbouring rows, rows short of a slice,
rows without some or all of the diagonals, rows with other columns, unsorted
and repeated columns, one level and many, and host execution on page-locked and
pageable memory."""
import numpy as np
import pytest

import mpk_gb300 as M
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _odd(a, seed, other, empty, order):
    """Every `other`-th row with columns anywhere, every `empty`-th row empty,
    every `order`-th with its columns reversed and its first repeated."""
    rng = np.random.default_rng(seed)
    rows = [a.col[a.ptr[i]:a.ptr[i + 1]] for i in range(a.n)]
    for i in range(0, a.n, other):
        rows[i] = np.sort(rng.choice(a.n, size=1 + i % 13, replace=False)).astype(np.int32)
    for i in range(7, a.n, order):
        rows[i] = np.concatenate([rows[i][::-1], rows[i][:1]])
    for i in range(3, a.n, empty):
        rows[i] = rows[i][:0]
    ptr = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    return M.Csr(ptr, np.concatenate(rows).astype(np.int32), rng.normal(size=int(ptr[-1])))


CASES = {
    "mesh5": (lambda: M.Csr.laplacian(100, 97), 4),
    "mesh5_narrow": (lambda: M.Csr.laplacian(7, 5003), 3),      # all diagonals within the own rows
    "mesh9": (lambda: M.Csr.diffusion(211, 203, sigma=1.0, seed=1), 3),
    "mesh9_wide": (lambda: M.Csr.diffusion(3001, 40, sigma=1.0, seed=2), 2),
    "box7": (lambda: M.Csr.laplacian(41, 37, 43), 8),
    "box7_thin": (lambda: M.Csr.laplacian(11, 9, 1201), 5),
    "tiny": (lambda: M.Csr.laplacian(5, 5), 1),
    "few_slices": (lambda: M.Csr.laplacian(9, 11), 31),
    # several levels per exchange: all of them, and a short last block
    "deep5": (lambda: M.Csr.laplacian(60, 61), 7),
    "deep5_one_slice": (lambda: M.Csr.laplacian(31, 170), 5),
    "deep9": (lambda: M.Csr.diffusion(91, 33, sigma=1.0, seed=6), 8),
    "deep9_many": (lambda: M.Csr.diffusion(150, 301, sigma=1.0, seed=6), 11),
    "deep7": (lambda: M.Csr.laplacian(20, 21, 22), 5),
    "odd_rows": (lambda: _odd(M.Csr.laplacian(60, 61, 20), 3, 4001, 53, 2503), 4),
    "odd_rows_2d": (lambda: _odd(M.Csr.laplacian(150, 149), 4, 1999, 31, 1777), 5),
}


def _run(plan, x, n, k, pinned=False):
    import torch
    vv = torch.zeros((k + 1) * n, dtype=torch.float64, pin_memory=pinned).numpy()
    vv[:n] = x
    for _ in range(2):  # flags and rings carry on from call to call
        vv[n:] = -7
        plan.exec_host(vv)
    plan.close()
    return vv


@pytest.mark.parametrize("name", CASES)
@pytest.mark.parametrize("valued", [False, True])
@pytest.mark.parametrize("arith", [M.ARITH_FMA, M.ARITH_SEPARATE, M.ARITH_DF64])
def test_equals_general_wavefront(name, valued, arith, gpu):
    make, k = CASES[name]
    a = make()
    a = M.Csr(a.ptr, a.col, M.uniform(3, a.nnz) if valued else None)
    x = M.uniform(5, a.n)
    want = _run(M.Plan.wave(a, k, arith=arith, ctas_per_sm=32), x, a.n, k)
    got = _run(M.Plan.wave(a, k, arith=arith), x, a.n, k)
    assert got.tobytes() == want.tobytes()
    got = _run(M.Plan.wave(a, k, arith=arith), x, a.n, k, pinned=True)
    assert got.tobytes() == want.tobytes()


@pytest.mark.parametrize("name", CASES)
@pytest.mark.parametrize("vt", [M.VALUE_F32, M.VALUE_BF16])
def test_mixed_bitwise_vs_fp32_oracle(name, vt, gpu):
    import torch
    make, k = CASES[name]
    a = make()
    val = M.uniform(7, a.nnz)
    if vt == M.VALUE_BF16:
        val = (val.astype(np.float32).view(np.uint32) & 0xFFFF0000).view(np.float32).astype(np.float64)
    a = M.Csr(a.ptr, a.col, val)
    plan = M.Plan.mixed(a, k, vt)
    e, _ = plan.mixed_scale()
    x = M.uniform(9, a.n).astype(np.float32)
    d = torch.zeros((k + 1) * a.n, dtype=torch.float32, device="cuda")
    d[:a.n] = torch.from_numpy(x).cuda()
    torch.cuda.synchronize()
    for _ in range(2):
        plan.exec_mixed_device(d.data_ptr())
        plan.sync()
    got = d.cpu().numpy().reshape(k + 1, a.n)
    want = O.spmm_f32(a.ptr, a.col, (a.val * 2.0 ** -e).astype(np.float32), x[:, None], k)[:, :, 0]
    tiny = np.finfo(np.float32).tiny  # scaled sums and scaled values round alike above the subnormal range
    fine = np.abs(want) >= 64 * tiny
    assert np.array_equal(got[fine], want[fine])
    assert np.all(np.abs(got[~fine]) < 128 * tiny)
