"""Waits that run out where copies into shared memory are under way: host
execution of the diagonal wavefront with matrix values (every form and mode of
it), and the packed batch with its matrix streamed and in shared memory.  The
call ends with ETIMEOUT, and the same plan then gives the oracle's bits."""
import numpy as np
import pytest

import mpk_gb300 as M
from oracle import oracle as O

pytestmark = pytest.mark.gpu

MATS = {
    "deep": lambda: M.Csr.laplacian(100, 97),
    "all": lambda: M.Csr.diffusion(400, 401, 1, sigma=0.5, seed=1),
    "pair": lambda: M.Csr.laplacian(64, 63, 40),
}


@pytest.mark.parametrize("name", MATS)
@pytest.mark.parametrize("valued", [False, True])
@pytest.mark.parametrize("arith", [M.ARITH_FMA, M.ARITH_DF64])
def test_host_execution(name, valued, arith, gpu):
    import torch
    a, k = MATS[name](), 5
    a = M.Csr(a.ptr, a.col, M.uniform(3, a.nnz) if valued else None)
    x = M.uniform(4, a.n)
    vv = torch.zeros((k + 1) * a.n, dtype=torch.float64, pin_memory=True).numpy()
    vv[:a.n] = x
    M.Plan.wave(a, k, arith=arith).exec_host(vv)
    want = vv.copy()
    if arith == M.ARITH_FMA:
        assert want.tobytes() == O.mpk(a.ptr, a.col, a.val, x, k, O.MODE_FMA).tobytes()
    plan = M.Plan.wave(a, k, arith=arith)
    plan.debug_stall(100)
    with pytest.raises(M.MpkError) as e:
        plan.exec_host(vv)
    assert e.value.code == M.ETIMEOUT
    plan.debug_stall(0)
    vv[a.n:] = -1
    plan.exec_host(vv)
    assert vv.tobytes() == want.tobytes()


@pytest.mark.parametrize("n", [700, 60000])  # the matrix in shared memory, streamed
@pytest.mark.parametrize("mode", [M.BATCH_STAGED, M.BATCH_STAGED4])
def test_packed_batch(n, mode, gpu):
    mats = [M.Csr.banded(n + 40 * q, 64, 5, 30, seed=q) for q in range(6)]
    total, nrhs, k = sum(m.n for m in mats), 16, 4
    X = M.uniform(9, total * nrhs).astype(np.float32).reshape(total, nrhs)
    vb = np.zeros((k + 1, total, nrhs), dtype=np.float32)
    vb[0] = X
    plan = M.Plan.batch(mats, nrhs, k, tune=mode)
    plan.debug_stall(100)
    with pytest.raises(M.MpkError) as e:
        plan.exec_batch_host(vb)
    assert e.value.code == M.ETIMEOUT
    plan.debug_stall(0)
    for _ in range(2):
        vb[1:] = -1
        plan.exec_batch_host(vb)
        r = 0
        for m in mats:
            want = O.spmm_f32(m.ptr, m.col, m.val.astype(np.float32), X[r:r + m.n], k)
            assert vb[:, r:r + m.n].tobytes() == want.tobytes()
            r += m.n
