"""s-step CG where basis values leave the range that the Gram's FP32 products
cover: columns scaled far down and far up, a right-hand side that is zero but
for one entry (its basis decays to nothing within a tile), every number of
columns, and a last tile that is not full.  The FP64 and double-float Gram
give solutions that agree, to what the solve's tolerance leaves."""
import numpy as np
import pytest

import mpk_gb300 as M
from mpk_gb300 import shifts as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(33, 31, 1), (16, 16, 9), (64, 64, 8)])
@pytest.mark.parametrize("s", [1, 4, 8, 10])
def test_gram_widths(dims, s, gpu):
    a = M.Csr.diffusion(*dims, sigma=0.5, dominance=0.1, seed=3)
    b = M.uniform(4, a.n)
    x, info = M.sstep_cg(a, b, s, shifts=S.from_lanczos(a, s), tol=1e-10)
    want, _ = M.cg(a, b, tol=1e-12)
    assert info["converged"]
    assert np.linalg.norm(x - want) / np.linalg.norm(want) < 1e-8


@pytest.mark.parametrize("factor", [1e-4, 1.0, 30.0])
def test_scaled_columns_and_point_source(factor, gpu):
    """scale = factor * the usual one: the columns grow or shrink by 1/factor
    each, over and past the range of one tile's FP32 products."""
    a = M.Csr.diffusion(48, 47, 1, sigma=0.5, dominance=0.2, seed=6)
    b = np.zeros(a.n)
    b[a.n // 2] = 1.0
    _, _, ghi = M.features(a)
    x, info = M.sstep_cg(a, b, 4, scale=factor * ghi / 2, tol=1e-9)
    want, _ = M.cg(a, b, tol=1e-12)
    assert info["converged"]
    assert np.linalg.norm(x - want) / np.linalg.norm(want) < 1e-7
