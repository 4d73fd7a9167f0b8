"""A kernel lets its successor start (pdl_trigger) with its last tile or group, never at once: the successor's CTAs wait
with their registers and shared memory held.  Checked on the sources: every call stands in the body of a loop over the
kernel's work, behind a condition on what is left of it."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dgkernel_b200", "csrc")
FILES = sorted(f for f in os.listdir(CSRC) if f.endswith(".cu") and "pdl_trigger()" in open(os.path.join(CSRC, f)).read())


@pytest.mark.parametrize("name", FILES)
def test_trigger_stands_behind_the_end_of_the_work(name):
    src = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
    calls = [ln for ln in src.splitlines() if "pdl_trigger()" in ln]
    assert calls
    for ln in calls:
        assert re.search(r"if \(.*(>=|!has1).*\) pdl_trigger\(\);", ln), f"{name}: {ln.strip()}"
