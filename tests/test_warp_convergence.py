"""A warp collective names the lanes that take part and every one of them has
to reach it.  `collective == x && collective == y` leaves the second out in the
lanes whose first comparison failed, while the others wait for them there."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cpvs_gb300", "csrc")
CALL = re.compile(r"__(?:shfl\w*|match_\w+|ballot|any|all|reduce_\w+)_sync\((?:[^()]|\((?:[^()]|\([^()]*\))*\))*\)")
SKIPPED = re.compile(r"COLLECTIVE[^;,{}]*(?:&&|\|\|)[^;,{}]*COLLECTIVE")


def skipped_collectives(text):
    text = re.sub(r"//[^\n]*", "", text)
    return [m.group(0) for m in SKIPPED.finditer(CALL.sub("COLLECTIVE", text))]


def test_the_search_finds_what_it_is_for():
    assert skipped_collectives("s = __shfl_sync(a, m, (int)l) == m && __shfl_sync(a, j, (int)l) == j;")
    assert not skipped_collectives("a = __ballot_sync(f, q && s), b = __ballot_sync(f, q && !s);")
    assert not skipped_collectives("s &= __shfl_sync(a, m, l) == m; s &= __shfl_sync(a, j, l) == j && s;")


@pytest.mark.parametrize("name", sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh"))))
def test_no_collective_behind_anothers_result(name):
    with open(os.path.join(CSRC, name)) as f:
        assert skipped_collectives(f.read()) == []
