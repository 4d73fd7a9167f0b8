"""The mixed stage's form with a matrix row per thread on problems of some size: the bits of the form with an element per
lane in both volume forms (a product merged with the subtraction after it shows in a few values of a hundred thousand
elements)."""
import numpy as np
import pytest

from dgkernel_b200.burgers import MIXED, BurgersProblem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("conservative", [0, 1])
@pytest.mark.parametrize("N,n,slabs", [(1, 40, 8), (2, 24, 1), (2, 33, 11), (3, 16, 16), (4, 13, 1)])
def test_bits(N, n, slabs, conservative):
    row = BurgersProblem(N, n, slabs, MIXED, "modes", conservative=conservative)
    lane = BurgersProblem(N, n, slabs, MIXED, "modes", conservative=conservative, warps=11)
    for p in (row, lane):
        p.run_stages(20)
    assert np.array_equal(row.get("u"), lane.get("u")) and np.array_equal(row.get("resu"), lane.get("resu"))
    assert np.isfinite(row.get("u")).all()
    for p in (row, lane):
        p.free()
