"""The tuner times the operator's own launch choice as one candidate and every slot shape once, and does not take a cached
number of warps that was timed as another form."""
import json

from dgkernel_b200 import autotune as T


def test_candidates_are_distinct_kernels():
    own = [c for c in T.MIXED_CANDIDATES if c["warps"] is None]
    assert own == [T.DEFAULT_SHAPE]
    # 11 warps and a full ring is what the operator chooses by itself where the row form is not taken
    assert {(c["warps"], c["ring"]) for c in T.MIXED_CANDIDATES} == {(None, None), (11, 6), (8, None), (8, 6), (4, None),
                                                                     (4, 6)}


def test_entries_without_the_own_choice_are_timed_again():
    def entry(best, times):
        return {"best": best, "ms_per_stage": {json.dumps(c, sort_keys=True): 1.0 for c in times}}
    old = [{"warps": w, "ring": r, "mma": False} for w in (11, 8, 4) for r in (None, 6)]
    assert not T.current(entry({"warps": 8, "ring": None, "mma": False}, old))
    assert T.current(entry({"warps": 8, "ring": 6, "mma": False}, old))
    assert T.current(entry({"warps": 8, "ring": None, "mma": True}, old))
    for c in T.MIXED_CANDIDATES:
        assert T.current(entry(c, T.MIXED_CANDIDATES))
