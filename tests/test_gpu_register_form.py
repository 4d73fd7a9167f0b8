"""The register-staged form of the plain stage (DGK_DISABLE_TMA=1 when the operator is built; orders 1..5) against the
FP64 oracle: the bounds of the parity tests, 1e-12 in FP64 and 2e-5 in FP32, after 5 stages, with partitions that are not a
multiple of its tiles.  The switch concerns the stage of these orders alone: the compact form is refused under it."""
import numpy as np
import pytest

import dgkernel_b200 as d
from dgkernel_b200.burgers import BurgersProblem
from oracle import burgers_ref as b
from oracle import oracle as O

from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,tol", [(np.float64, 1e-12), (np.float32, 2e-5)])
@pytest.mark.parametrize("N,n,nslab", [(1, 6, 3), (2, 4, 2), (3, 3, 3), (4, 3, 1), (5, 3, 3)])
def test_against_oracle(N, n, nslab, dtype, tol, monkeypatch):
    monkeypatch.setenv("DGK_DISABLE_TMA", "1")
    cons = N % 2
    P = BurgersProblem(N, n, nslab, dtype, "modes", conservative=cons)
    P.dt /= 4
    u = P.u0.astype(np.float64)
    O.RunState(b.Problem(N, n, nslab, "sine")).run(u, np.zeros_like(u), P.dt, 5, conservative=cons, threads=4)
    P.run_stages(5)
    assert rel_l2(P.get("u"), u) < tol
    P.free()


def test_compact_needs_the_copies(monkeypatch):
    monkeypatch.setenv("DGK_DISABLE_TMA", "1")
    with pytest.raises(d.DGKError, match="compact=1"):
        BurgersProblem(2, 4, 2, np.float64, "modes", compact=True)
