"""Device memory of wavefront plans (host code against the runtime of
fake_cudart.c): what a plan says it holds is what it holds, the diagonal
wavefront holds no more than the general one, and nothing is left behind."""
import pytest

import fake_cudart


@pytest.mark.parametrize("valued", [False, True])
@pytest.mark.parametrize("arith", ["FMA", "SEPARATE", "DF64"])
@pytest.mark.parametrize("mesh", ["M.Csr.laplacian(40, 41, 42)", "M.Csr.diffusion(200, 201, 1, sigma=0.5, seed=1)"])
def test_no_more_than_the_general_wavefront(mesh, arith, valued, tmp_path):
    fake_cudart.run(str(tmp_path), f"""
a = {mesh}
a = a if {valued} else a.pattern()
held = []
for ctas in (0, 32):
    p = M.Plan.wave(a, 4, arith=M.ARITH_{arith}, ctas_per_sm=ctas)
    held.append(live())
    assert live() == p.info()["device_bytes"], (live(), p.info())
    p.close()
    assert live() == 0
assert held[0] <= held[1], held
""")


@pytest.mark.parametrize("mode", ["DEFAULT", "TUNE"])
def test_batch_takes_the_csr_kernel_where_the_packed_matrix_finds_no_memory(mode, tmp_path):
    """Rows of one entry take twice their CSR bytes when packed; a plan that
    has a choice of kernels is made of those that fit, and refused where none does."""
    fake_cudart.run(str(tmp_path), f"""
n = 200000
i = np.arange(n, dtype=np.int32)
mats = [M.Csr(np.arange(n + 1, dtype=np.int32), i[::-1].copy() if q else i, np.ones(n)) for q in range(2)]
vectors = 3 * 2 * n * 4 * 4 if "{mode}" == "TUNE" else 0
p = M.Plan.batch(mats, 4, 2, tune=M.BATCH_STAGED)
packed = live()
p.close()
csr = 2 * n * 12
assert packed > csr + 1000000
fake.fake_limit(csr + 500000)
raises(M.ECUDA, lambda: M.Plan.batch(mats, 4, 2, tune=M.BATCH_STAGED))
fake.fake_limit(csr + 500000 + vectors)
p = M.Plan.batch(mats, 4, 2, tune=M.BATCH_{mode})
assert not p.batch_info()["staged"] and live() == p.batch_info()["device_bytes"]
p.exec_batch_device(1 << 20)
p.close()
fake.fake_limit(csr // 2 + vectors)
assert live() == 0
try:
    M.Plan.batch(mats, 4, 2, tune=M.BATCH_{mode})
    raise AssertionError("no error")
except M.MpkError as e:
    assert e.code in (M.ECUDA, M.ENOMEM) and str(e)
assert live() == 0
""")
