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
