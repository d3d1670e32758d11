"""Device memory that a call or a plan clears or fills is ready before any
kernel can read it.  cudaMemset, and cudaMemcpy from pageable or device memory,
work on the legacy default stream and may return before the device has done
them, while plans and callers launch on streams that do not wait for that one:
between them and the next launch, or the return to the caller, something must
wait."""
import pytest

import fake_cudart

PLANS = {
    "batch_tune": "M.Plan.batch(B, 4, 2, tune=M.BATCH_TUNE)",
    "batch_tune_2": "M.Plan.batch(B, 2, 2, tune=M.BATCH_TUNE)",
    "batch_default": "M.Plan.batch(B, 4, 2, tune=M.BATCH_DEFAULT)",
    "batch_staged": "M.Plan.batch(B, 4, 2, tune=M.BATCH_STAGED2)",
    "wave": "M.Plan.wave(A, 3)",
    "wave_fixed": "M.Plan.wave(A.pattern(), 3, arith=M.ARITH_FIXED)",
    "pipe": "M.Plan.pipe(A, 3)",
    "spmv": "M.Plan.spmv(A, 3)",
    "mixed": "M.Plan.mixed(V, 3)",
    "mixed_tiles": "M.Plan.mixed_tiles(V, M.partition_rcb(A.coords, 4), 4, 3)",
}
SETUP = """
A = M.Csr.laplacian(40, 41)
V = M.Csr.diffusion(40, 41, 1, sigma=0.5, seed=1)
B = [M.Csr.banded(300 + 50 * q, 16, 3, 9, seed=q) for q in range(3)]
"""


def _check(log):
    """Follows the legacy stream: what is pending on it at each launch on another stream and at each mark."""
    pending = None
    for w in log:
        if w[-1] == "legacy" and (w[0] == "memset" or w[0] == "memcpy" and w[1] in ("1", "3")):  # up, or on the device
            pending = w
        elif w[0] == "memcpy" and w[3] == "legacy" or w[0] == "sync" and w[1] in ("legacy", "device"):
            pending = None
        elif w[0] == "mark" or w[0] == "launch" and w[5] != "(nil)":
            assert pending is None, (pending, w)


@pytest.mark.parametrize("plan", PLANS)
def test_cleared_before_the_plan_is_used(plan, tmp_path):
    log = fake_cudart.run(str(tmp_path), SETUP + f"""
p = {PLANS[plan]}
mark("returned")
""")
    assert log[-1] == ["mark", "returned"]
    _check(log)


@pytest.mark.parametrize("plan", ["batch_default", "batch_staged", "pipe", "wave", "mixed"])
def test_cleared_before_the_call_after_a_timeout(plan, tmp_path):
    """The status, flags and counters that a device-side time-out leaves."""
    log = fake_cudart.run(str(tmp_path), SETUP + f"""
p = {PLANS[plan]}
fake.fake_status(2)
mark("sync")
raises(M.ETIMEOUT, p.sync)
mark("returned")
""")
    at = log.index(["mark", "sync"])
    assert any(w[0] == "memset" for w in log[at:])
    _check(log)


@pytest.mark.parametrize("basis", ["M.SSTEP_BASIS_MPK", "M.SSTEP_BASIS_STEPS"])
def test_solve_starts_from_what_it_uploaded(basis, tmp_path):
    """The solver's own stream, up to the point where the fake runtime has no graphs."""
    log = fake_cudart.run(str(tmp_path), SETUP + f"""
try: M.sstep_cg(V, np.ones(V.n), 4, scale=1.0, basis={basis})
except M.MpkError: pass
mark("returned")
""")
    assert any(w[0] == "launch" for w in log)
    _check(log)
