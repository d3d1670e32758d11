"""The diagonal wavefront's layouts (host code only)."""
import numpy as np
import pytest

import diag_probe as D
import fake_cudart
import mpk_gb300 as M


@pytest.mark.parametrize("make,form", [(lambda: M.Csr.laplacian(160, 160, 140), D.FMA),
                                       (lambda: M.Csr.diffusion(1600, 1601, 1, sigma=0.5, seed=1), D.DF_VAL),
                                       (lambda: M.Csr.diffusion(2048, 2200, 1, sigma=0.5, seed=1), D.F32)])
def test_too_large_is_known_before_the_rows_are_read(make, form):
    """A matrix beyond the shared memory of all the SMs is turned away by its sizes alone."""
    got = D.layout(make(), form, 4)
    assert not got["fits"] and got["w"] > 0 and got["scanned"] == 0


def _with_rows(a, rows, near, length=7):
    """`a` with `length` columns anywhere (or within `near`) in the given rows."""
    rng = np.random.default_rng(3)
    cols = [a.col[a.ptr[i]:a.ptr[i + 1]] for i in range(a.n)]
    for i in rows:
        c = rng.integers(0, a.n, length) if near is None else i + rng.integers(-near, near, length)
        cols[i] = np.unique(np.clip(c, 0, a.n - 1)).astype(np.int32)
    ptr = np.concatenate([[0], np.cumsum([len(c) for c in cols])]).astype(np.int32)
    return M.Csr(ptr, np.concatenate(cols).astype(np.int32))


IRREGULAR = {  # rows, columns within, and in which forms the layout is the faster
    "none": (lambda n: [], None, (D.FMA, D.SEP_VAL, D.DF, D.F32)),
    "scattered": (lambda n: range(5, n, 32 * 25), None, (D.FMA, D.SEP_VAL, D.DF, D.F32)),
    "block": (lambda n: range(n // 100), None, ()),
    "near_block": (lambda n: range(n // 25), 3000, ()),
    "one_block_full": (lambda n: range(8736 * 3, 8736 * 3 + 32 * 200), 3000, ()),
    "one_slice": (lambda n: range(32 * 500, 32 * 501), 3000, (D.FMA, D.SEP_VAL, D.DF, D.F32)),
}


@pytest.mark.parametrize("name", IRREGULAR)
@pytest.mark.parametrize("form", [D.FMA, D.SEP_VAL, D.DF, D.F32])
def test_irregular_rows_where_they_cost_less_than_they_gain(name, form):
    rows, near, faster = IRREGULAR[name]
    a = M.Csr.laplacian(110, 110, 110)
    got = D.layout(_with_rows(a, rows(a.n), near), form, 5)
    assert bool(got["fits"]) == (form in faster), got


def test_irregular_rows_on_small_meshes():
    """Few slices a block: any row that runs entry by entry is the longest of its level."""
    a = M.Csr.laplacian(100, 100)
    assert D.layout(a, D.FMA, 5)["fits"] and D.layout(a, D.FMA, 5)["mode"] == D.DEEP
    for form in (D.FMA, D.SEP, D.DF):
        assert not D.layout(_with_rows(a, [4321], None), form, 5)["fits"]


@pytest.mark.parametrize("make", ["M.Csr.diffusion(120, 110, 1, sigma=0.5, seed=1)", "M.Csr.diffusion(40, 41, 42, sigma=0.5, seed=1)"])
@pytest.mark.parametrize("vt,form", [("F32", D.F32), ("BF16", D.BF16)])
def test_mixed_plans_count_the_rows_they_compute(make, vt, form, tmp_path):
    """With several levels per exchange a block computes rows of its neighbours too."""
    a = eval(make)
    rows = D.layout(a, form, 8)["rows"]
    assert rows > 8 * a.n or a.n > 20000
    fake_cudart.run(str(tmp_path), f"""
p = M.Plan.mixed({make}, 8, M.VALUE_{vt})
assert p.info()["rows_computed"] == {rows}, (p.info(), {rows})
""")
