"""Marking an active element's neighbours in the composite's sensor pass on a mesh of many partitions: a neighbour's slot is
found by a walk over the partitions, one walk per lane and face.  With every element active, order 1, 48^3 x 6, the pass
in 48 partitions may take 2.75 times as long as in one: measured 1.95 with a walk per lane, 3.9 with an element's four
walks one after the other.  Device time by the profiler, in a process of its own."""
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

TIMED = """
import torch
from torch.profiler import ProfilerActivity, profile
from dgkernel_b200 import sensor as SN
from dgkernel_b200.burgers import MIXED, BurgersProblem
torch.zeros(1, device="cuda")
for slabs in (1, 48):
    P = BurgersProblem(1, 48, slabs, MIXED, "modes", mma=True, learned="mlp", conf=(0.5, 0.5))
    P.dt = 1e-9
    P.set_sensor("mlp", SN.init_params(P.el.Np, seed=3))  # outputs near one half: every element has viscosity
    P.run_stages(10)
    P.runner.Sync()
    with profile(activities=[ProfilerActivity.CUDA]) as pr:
        P.run_stages(20)
        P.runner.Sync()
    ev, = [e for e in pr.key_averages() if "ls_sensor_kernel" in e.key]
    print("TIME", ev.device_time_total / ev.count)
    P.free()
"""


def test_marking_in_many_partitions():
    out = subprocess.run([sys.executable, "-c", TIMED], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr
    one, many = [float(ln.split()[1]) for ln in out.stdout.splitlines() if ln.startswith("TIME")]
    print(f"sensor pass: {one:.1f} us in one partition, {many:.1f} us in 48")
    assert many < 2.75 * one
