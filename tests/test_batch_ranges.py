"""Row ranges of a batch's thread blocks, from what a plan uploads: the CSR
kernel spreads every batch evenly over all its blocks, however small."""
import pytest

import fake_cudart

MATS = {
    "one": "[M.Csr.banded(40000, 64, 5, 30, seed=1)]",
    "few": "[M.Csr.banded(300 + 500 * q, 64, 5, 30, seed=q) for q in range(6)]",
    "many": "[M.Csr.banded(50 + q, 16, 5, 20, seed=q) for q in range(300)]",
    "tiny": "[M.Csr.banded(40 + q, 2, 1, 2, seed=q) for q in range(20)]",
}


@pytest.mark.parametrize("mats", MATS)
@pytest.mark.parametrize("nrhs", [1, 2])
def test_csr_kernel_takes_all_blocks(mats, nrhs, tmp_path):
    fake_cudart.run(str(tmp_path), f"""
mats = {MATS[mats]}
p = M.Plan.batch(mats, {nrhs}, 3, tune=M.BATCH_DEFAULT)
i = p.batch_info()
assert not i["staged"] and i["ngroup"] == 1
lo = upload(i["grid"] + 1, np.int32, back=1)  # before the dependencies, which are as many
ptr = np.concatenate([[0], np.cumsum(np.concatenate([np.diff(m.ptr) for m in mats]))])
assert lo[0] == 0 and lo[-1] == len(ptr) - 1 and np.all(np.diff(lo) >= 0)
share, longest = np.diff(ptr[lo]), np.diff(ptr).max()
assert share.max() <= ptr[-1] / i["grid"] + longest
""")
