"""Which kernel a call launches, and with what of the device, by the rules of
its plan (host code against the runtime of fake_cudart.c: 152 SMs)."""
import pytest

import fake_cudart


def _kernels(log, name):
    return [w for w in fake_cudart.launches(log) if name in w[0]]


@pytest.mark.parametrize("n,ints", [(256 * 152, False), (256 * 152 + 1, True)])
@pytest.mark.parametrize("arith,code", [("SEPARATE", 1), ("FMA", 0)])
def test_spmv_integer_products_where_the_fp64_pipe_is_busy(n, ints, arith, code, tmp_path):
    log = fake_cudart.run(str(tmp_path), f"""
a = M.Csr.banded({n}, 8, 2, 4, seed=1)
p = M.Plan.spmv(a, 3, arith=M.ARITH_{arith})
p.exec_host(np.zeros(4 * a.n))
""")
    got = _kernels(log, "spmv_level_kernel")
    want = f"spmv_level_kernelILi{code}ELb1ELb{int(ints and arith == 'SEPARATE')}E"
    assert len(got) == 3 and all(want in w[0] for w in got), got


@pytest.mark.parametrize("make,k,most", [
    ("M.Plan.wave(M.Csr.laplacian(100, 100).pattern(), 4)", 4, 20000),
    ("M.Plan.wave(M.Csr.laplacian(100, 100), 4, arith=M.ARITH_DF64)", 4, 60000),
    ("M.Plan.wave(M.Csr.laplacian(60, 60, 60).pattern(), 4)", 4, 40000),
    ("M.Plan.wave(M.Csr.laplacian(128, 128, 128).pattern(), 4)", 4, 231424),
])
def test_diagonal_wavefront_takes_the_shared_memory_it_needs(make, k, most, tmp_path):
    """A small plan leaves room on every SM, so that plans on several streams run side by side."""
    log = fake_cudart.run(str(tmp_path), f"""
p = {make}
p.exec_host(np.zeros({k + 1} * p.n))
""")
    (kernel, blocks, threads, smem, _), = _kernels(log, "diag_kernel")
    assert blocks <= 152 and smem <= most


def test_small_batch_takes_the_shared_memory_it_needs(tmp_path):
    log = fake_cudart.run(str(tmp_path), """
mats = [M.Csr.banded(300 + 500 * q, 64, 5, 30, seed=q) for q in range(6)]
for mode in (M.BATCH_DEFAULT, M.BATCH_STAGED, M.BATCH_STAGED4):
    p = M.Plan.batch(mats, 4, 3, tune=mode)
    i = p.batch_info()
    print(i["grid"], i["window_bytes"])
    p.exec_batch_host(np.zeros((4, sum(m.n for m in mats), 4), dtype=np.float32))
""")
    info = [tuple(map(int, line.split())) for line in open(tmp_path / "out.txt")]
    got = _kernels(log, "batch_pack_kernel")
    assert [(w[1], w[3]) for w in got] == info
    for kernel, blocks, threads, smem, _ in got:
        assert smem <= threads * 150  # of about 225 bytes a thread


@pytest.mark.parametrize("make,kind", [
    ("M.Csr.laplacian(140, 140, 138)", 1),  # columns near, the levels in L2
    ("M.Csr.laplacian(150, 150, 151)", 0),  # beyond L2
    ("M.Csr.laplacian(240, 240, 3)", 0),    # columns beyond 16 bits
    ("M.Csr.diffusion(300, 301, 1, sigma=0.5, seed=1)", 1),
])
def test_general_wavefront_takes_integer_products_where_the_fp64_pipe_is_busy(make, kind, tmp_path):
    log = fake_cudart.run(str(tmp_path), f"""
a = {make}.pattern()
p = M.Plan.wave(a, 1, ctas_per_sm=32)
p.exec_device(1 << 20)
""")
    (kernel, *_), = _kernels(log, "wave_kernel")
    assert f"Li{kind}EEEv" in kernel, kernel


@pytest.mark.parametrize("entries,valued,arith,code,kind", [
    (8, True, "FMA", 0, 1), (9, True, "FMA", 0, 3), (28, True, "SEPARATE", 1, 2), (29, True, "SEPARATE", 1, 3),
    (29, False, "SEPARATE", 1, 1), (28, False, "SEPARATE", 1, 2), (8, True, "SEPARATE", 1, 2), (29, True, "FMA", 0, 3),
])
def test_general_wavefront_goes_over_rows_by_their_average_length(entries, valued, arith, code, kind, tmp_path):
    log = fake_cudart.run(str(tmp_path), f"""
a = M.Csr.banded(5000, 128, {entries}, {entries}, seed=1)
p = M.Plan.wave(a if {valued} else a.pattern(), 1, arith=M.ARITH_{arith})
p.exec_device(1 << 20)
""")
    (kernel, *_), = _kernels(log, "wave_kernel")
    assert f"wave_kernelILi{code}ELb{int(valued)}E" in kernel and f"Li{kind}EEEv" in kernel, kernel


@pytest.mark.parametrize("nx,length,long", [(100, 64, False), (100, 65, True), (300, 200, True), (2000, 65, False)])
@pytest.mark.parametrize("arith,code", [("SEPARATE", 1), ("FMA", 0)])
def test_general_wavefront_with_one_long_row(nx, length, long, arith, code, tmp_path):
    log = fake_cudart.run(str(tmp_path), f"""
a = M.Csr.laplacian({nx}, {nx})
i = a.n // 2
ptr, cut = a.ptr.astype(np.int64), slice(a.ptr[i], a.ptr[i + 1])
col = np.concatenate([a.col[:cut.start], np.arange(i - 30, i - 30 + {length}), a.col[cut.stop:]])
ptr[i + 1:] += {length} - (cut.stop - cut.start)
a = M.Csr(ptr.astype(np.int32), col.astype(np.int32), np.ones(len(col)))
p = M.Plan.wave(a, 1, arith=M.ARITH_{arith}, ctas_per_sm=32)
p.exec_device(1 << 20)
""")
    (kernel, *_), = _kernels(log, "wave_kernel")
    assert f"wave_kernelILi{code}ELb1E" in kernel and ("Li3EEEv" in kernel) == long, kernel
