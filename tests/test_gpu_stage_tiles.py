"""Plain FP64 and FP32 stages on partitions that start on any value (a tile's bulk copies start on the 16 bytes that hold
its first value) and end inside a tile: the bits of the one-partition run, since an element's arithmetic does not depend
on its tile; and the FP32 stage against the FP64 one within the FP32 bound of the oracle tests (2e-5), every order."""
import numpy as np
import pytest

from dgkernel_b200 import mesh as M
from dgkernel_b200._lib import check, lib
from dgkernel_b200.burgers import BurgersProblem, _TetBurgers, _pd, random_modes

from conftest import rel_l2

pytestmark = pytest.mark.gpu


class _Parts(_TetBurgers):
    """A periodic n^3 x 6 problem whose partitions are element ranges of the given sizes."""

    def __init__(self, N, n, sizes, dtype, conservative):
        VX, VY, VZ, EToV, EToVp, _ = M.kuhn_mesh(n, 1)
        EToE, EToF = M.ti_connect3d(EToVp)
        EToP = np.repeat(np.arange(len(sizes), dtype=np.int64), sizes)
        self._assemble(N, VX, VY, VZ, EToV, EToE, EToF, EToP, sizes, dtype, None)
        r, modes = self.runner, random_modes(7)
        check(lib().dgk_init_field(r._h, b"u", b"X", b"Y", b"Z", 2, 0.5, 0.0, len(modes), _pd(modes)), r._h)
        self._finish(0.3, conservative)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("N,sizes", [(1, (33, 1, 128)), (2, (17, 145)), (3, (9, 16, 137)), (4, (7, 15, 17, 123)),
                                     (4, (1, 161)), (5, (3, 16, 143)), (6, (5, 157)), (7, (8, 9, 145))])
def test_partition_starts(N, sizes, dtype):
    cons = N % 2
    one = BurgersProblem(N, 3, 1, dtype, "modes", seed=7, conservative=cons)
    cut = _Parts(N, 3, list(sizes), dtype, cons)
    assert np.array_equal(cut.get("u"), one.get("u"))
    for p in (one, cut):
        p.dt = one.dt
        p.run_stages(7)
    assert np.array_equal(cut.get("u"), one.get("u")) and np.array_equal(cut.get("resu"), one.get("resu"))
    for p in (one, cut):
        p.free()


@pytest.mark.parametrize("conservative", [0, 1])
@pytest.mark.parametrize("N,n,slabs", [(1, 9, 9), (2, 8, 4), (3, 7, 7), (4, 9, 3), (5, 6, 2), (6, 5, 5), (7, 4, 1)])
def test_fp32_tracks_fp64(N, n, slabs, conservative):
    a = BurgersProblem(N, n, slabs, np.float64, "modes", seed=7, conservative=conservative)
    b = BurgersProblem(N, n, slabs, np.float32, "modes", seed=7, conservative=conservative)
    a.dt = b.dt = a.dt / 10
    for p in (a, b):
        p.run_stages(10)
    assert rel_l2(b.get("u"), a.get("u")) < 2e-5
    for p in (a, b):
        p.free()
