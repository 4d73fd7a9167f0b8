"""The mixed stage's slot form (an element per lane) on problems small enough for the form with a matrix row per thread:
an explicit number of warps selects it, and with its ring as deep as shared memory allows it tracks the FP64 oracle
within the mixed stage's bound (1e-7 over 10 stages) and gives the row form's bits."""
import subprocess
import sys

import numpy as np
import pytest

from dgkernel_b200.burgers import MIXED, BurgersProblem
from oracle import burgers_ref as b
from oracle import oracle as O

from conftest import ROOT, rel_l2

pytestmark = pytest.mark.gpu

SEEN = """
import sys, torch
from torch.profiler import ProfilerActivity, profile
from dgkernel_b200.burgers import MIXED, BurgersProblem
torch.zeros(1, device="cuda")
for kw in ({}, {"warps": 8}, {"ring": 4}, {"warps": 11}):
    P = BurgersProblem(3, 4, 1, MIXED, "modes", **kw)
    P.run_stages(2)
    P.runner.Sync()
    with profile(activities=[ProfilerActivity.CUDA]) as pr:
        P.run_stages(2)
        P.runner.Sync()
    names = " ".join(e.key for e in pr.key_averages())
    print("FORM", "rows" if "rhs_stage_rows" in names else "slots" if "rhs_stage_mixed" in names else names)
    P.free()
"""


def test_a_launch_shape_selects_the_slot_form():
    out = subprocess.run([sys.executable, "-c", SEEN], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr
    assert [ln.split()[1] for ln in out.stdout.splitlines() if ln.startswith("FORM")] == ["rows"] + ["slots"] * 3


@pytest.mark.parametrize("conservative", [0, 1])
@pytest.mark.parametrize("warps", [4, 8, 11])
@pytest.mark.parametrize("N,n,nslab", [(1, 5, 5), (2, 4, 2), (3, 5, 1), (4, 5, 5)])
def test_slot_form_with_a_full_ring(N, n, nslab, warps, conservative):
    P = BurgersProblem(N, n, nslab, MIXED, "modes", warps=warps, conservative=conservative)
    Q = BurgersProblem(N, n, nslab, MIXED, "modes", conservative=conservative)
    u = np.ascontiguousarray(P.u0, dtype=np.float64).copy()
    O.RunState(b.Problem(N, n, nslab, "sine")).run(u, np.zeros_like(u), P.dt, 10, conservative=conservative, threads=4)
    for p in (P, Q):
        p.run_stages(10)
    assert rel_l2(P.get("u"), u) < 1e-7
    assert np.array_equal(P.get("u"), Q.get("u")) and np.array_equal(P.get("resu"), Q.get("resu"))
    for p in (P, Q):
        p.free()
