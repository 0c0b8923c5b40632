"""Shared-key shape candidates (no GPU): none is timed twice under different names."""
import os
import re

from cumayo_b200 import autotune as AT

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_hash_sizes_only_where_they_have_an_effect():
    src = open(os.path.join(ROOT, "cumayo_b200", "csrc", "ops.h")).read()
    assert int(re.search(r"HASH_WARP_MAX = (\d+);", src).group(1)) == AT.HASH_WARP_MAX
    assert AT.shared_candidates(AT.HASH_WARP_MAX + 1) == AT.SHARED_CANDIDATES
    for batch in (1, 301, AT.HASH_WARP_MAX):
        few = AT.shared_candidates(batch)
        assert {(g, p) for _, g, p in few} == {(g, p) for _, g, p in AT.SHARED_CANDIDATES}
        assert len(few) == len({(g, p) for _, g, p in few})
