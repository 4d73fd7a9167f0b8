"""Mixed stage with a matrix row per thread (orders 1..4): tiles cut by ragged partitions give the bits of the
one-partition run (an element's arithmetic does not depend on its tile), and that run tracks the FP64 stage within the
mixed stage's bound (1e-7 over 10 stages)."""
import numpy as np
import pytest

from dgkernel_b200 import mesh as M
from dgkernel_b200._lib import check, lib
from dgkernel_b200.burgers import MIXED, BurgersProblem, _TetBurgers, _pd, random_modes

from conftest import rel_l2

pytestmark = pytest.mark.gpu


class _Parts(_TetBurgers):
    """A periodic n^3 x 6 problem whose partitions are element ranges of the given sizes."""

    def __init__(self, N, n, sizes, conservative):
        VX, VY, VZ, EToV, EToVp, _ = M.kuhn_mesh(n, 1)
        EToE, EToF = M.ti_connect3d(EToVp)
        EToP = np.repeat(np.arange(len(sizes), dtype=np.int64), sizes)
        self._assemble(N, VX, VY, VZ, EToV, EToE, EToF, EToP, sizes, MIXED, None)
        r, modes = self.runner, random_modes(7)
        check(lib().dgk_init_field(r._h, b"u", b"X", b"Y", b"Z", 2, 0.5, 0.0, len(modes), _pd(modes)), r._h)
        self._finish(0.3, conservative)


@pytest.mark.parametrize("conservative", [0, 1])
@pytest.mark.parametrize("N,sizes", [(1, (1, 64, 97)), (2, (31, 33, 98)), (3, (1, 12, 13, 136)), (4, (13, 14, 15, 120)),
                                     (4, (2, 160))])
def test_partial_tiles(N, sizes, conservative):
    one = BurgersProblem(N, 3, 1, MIXED, "modes", seed=7, conservative=conservative)
    ref = BurgersProblem(N, 3, 1, np.float64, "modes", seed=7, conservative=conservative)
    cut = _Parts(N, 3, list(sizes), conservative)
    assert np.array_equal(cut.get("u"), one.get("u"))
    for p in (one, ref, cut):
        p.dt = one.dt
        p.run_stages(10)
    assert np.array_equal(cut.get("u"), one.get("u"))
    assert rel_l2(one.get("u"), ref.get("u")) < 1e-7
    for p in (one, ref, cut):
        p.free()


@pytest.mark.parametrize("conservative", [0, 1])
@pytest.mark.parametrize("N,n,slabs", [(1, 5, 5), (2, 5, 1), (3, 6, 3), (4, 5, 5)])
def test_both_forms_give_the_same_bits(N, n, slabs, conservative):
    """A ring depth asks for the form with an element per lane."""
    row = BurgersProblem(N, n, slabs, MIXED, "modes", seed=7, conservative=conservative)
    lane = BurgersProblem(N, n, slabs, MIXED, "modes", seed=7, conservative=conservative, ring=4)
    for p in (row, lane):
        p.run_stages(10)
    assert np.array_equal(row.get("u"), lane.get("u")) and np.array_equal(row.get("resu"), lane.get("resu"))
    for p in (row, lane):
        p.free()


def test_many_tiles_per_cta():
    """More tiles than the persistent grid holds, with a ragged tail in every partition."""
    one = BurgersProblem(3, 14, 1, MIXED, "modes", seed=7)
    ref = BurgersProblem(3, 14, 1, np.float64, "modes", seed=7)
    cut = BurgersProblem(3, 14, 14, MIXED, "modes", seed=7)
    for p in (one, ref, cut):
        p.run_stages(10)
    assert np.array_equal(cut.get("u"), one.get("u"))
    assert rel_l2(one.get("u"), ref.get("u")) < 1e-7
    for p in (one, ref, cut):
        p.free()
