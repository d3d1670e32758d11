"""The diagonal wavefront's layouts (host code only)."""
import numpy as np
import pytest

import diag_probe as D
import mpk_gb300 as M


@pytest.mark.parametrize("make,form", [(lambda: M.Csr.laplacian(160, 160, 140), D.FMA),
                                       (lambda: M.Csr.diffusion(1600, 1601, 1, sigma=0.5, seed=1), D.DF_VAL),
                                       (lambda: M.Csr.diffusion(2048, 2200, 1, sigma=0.5, seed=1), D.F32)])
def test_too_large_is_known_before_the_rows_are_read(make, form):
    """A matrix beyond the shared memory of all the SMs is turned away by its sizes alone."""
    got = D.layout(make(), form, 4)
    assert not got["fits"] and got["w"] > 0 and got["scanned"] == 0
