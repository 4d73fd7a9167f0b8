"""Kernels launched with programmatic dependent launch overlap the kernel before them, so a non-coherent load (__ldg,
ld.global.nc) may read only what no kernel writes between an operator's build and its launch: its constants.  Checked on
the sources: every such load in a file that launches this way names one of the arrays below, which the operators upload
when they are built."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dgkernel_b200", "csrc")
CONSTANTS = {"Dr", "Ds", "Dt", "LIFT", "Vinv", "rexp", "amat", "bmat", "D64", "L64", "bary", "vtx", "ftab", "fmask"}
FILES = sorted(f for f in os.listdir(CSRC) if f.endswith(".cu") and "launch_pdl(" in open(os.path.join(CSRC, f)).read())


def test_the_stage_kernels_are_among_them():
    assert {"rows.cu", "oz.cu", "mixed.cu", "tcm.cu", "av.cu", "lsens.cu", "kernels_tma.cu", "kernels_wide.cu"} <= set(FILES)


@pytest.mark.parametrize("name", FILES)
def test_non_coherent_loads_read_constants(name):
    src = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
    for m in re.finditer(r"__ldg\(\s*([^;]*)", src):
        arr = re.match(r"&?A\.(\w+)", m.group(1))
        assert arr and arr.group(1) in CONSTANTS, f"{name}: __ldg({m.group(1)[:60]}"
    # the one function around ld.global.nc loads matrix fragments: its arguments come from A.D64 and A.L64
    users = set(re.findall(r"(\w+)\(const double \*p\) \{\s*double v;\s*asm volatile\(\"ld\.global\.nc", src))
    assert len(re.findall(r"ld\.global\.nc", src)) == len(users)
    for f in users:
        for arg in re.findall(rf"= {f}\((\w+)", src):
            made = re.findall(rf"const double \*{arg} = A\.(\w+)", src)
            assert made and set(made) <= CONSTANTS, f"{name}: {f}({arg})"
    # a restrict-qualified pointer to const lets the compiler choose the non-coherent load by itself
    assert not re.search(r"const\s+\w+\s*\*\s*__restrict__", src), name
