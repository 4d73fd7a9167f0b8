"""The mixed stage's form with a matrix row per thread on problems of some size: the bits of the form with an element per
lane in both volume forms (a product merged with the subtraction after it shows in a few values of a hundred thousand
elements), also at order 2 beyond 1,300 elements per SM, where that form had been taken, and there a stage is the faster
one (measured 0.85 of it at 48^3 x 6, bound 0.95)."""
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


def _time(**kw):
    import torch
    st = torch.cuda.Stream()
    P = BurgersProblem(2, 48, 1, MIXED, "modes", stream=st.cuda_stream, **kw)
    P.dt = 1e-9
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    best = float("inf")
    for _ in range(5):
        with torch.cuda.stream(st):
            e0.record(st)
            P.run_stages(20)
            e1.record(st)
        e1.synchronize()
        best = min(best, e0.elapsed_time(e1))
    P.free()
    return best


def test_large_problems_take_the_faster_form():
    assert _time() < 0.95 * _time(warps=11)
