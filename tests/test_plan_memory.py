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
