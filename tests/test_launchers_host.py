"""An operator swaps its buffers after a launch, so a launcher that can decline must not be ignored: every call of a
launcher that returns bool is tested by the operator (the others throw)."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dgkernel_b200", "csrc")


def test_declined_launches_are_noticed():
    decl = re.findall(r"^bool (launch_\w+)\(", open(os.path.join(CSRC, "kernels.hpp")).read(), re.M)
    assert decl
    ops = open(os.path.join(CSRC, "ops.cu")).read()
    for name in decl:
        calls = re.findall(rf"([^\n]*)\b{name}(?:<\w+>)?\(", ops)
        assert calls, name
        for before in calls:
            assert before.rstrip().endswith("if (!"), f"{name}: its result is dropped after '{before.strip()}'"
