"""Bounded waits on the device, read from the sources: a warp that gives one up leaves as a whole.  Lanes count their polls each for itself; a lane
that left alone would be missing from the shuffles and barriers of the others, and a wait that ran out for lanes other than 0 only would
not be reported (lane 0 writes the error word)."""
import os
import re

import pytest

from tests.util import ROOT

CSRC = os.path.join(ROOT, "shadow-engine_b200", "csrc")
#: files whose kernels leave a loop or return where a wait of a whole warp ran out
FILES = ["sz_session_rows.cuh"]


def leaving_waits(text):
    """Statements `if (.. wait ..) {.. return / break ..}` -> the waits they call."""
    text = re.sub(r"//[^\n]*", "", text)
    for m in re.finditer(r"if \(([^;{}]*\bsz_mbar_wait\w*\([^;{}]*)\) *(\{[^{}]*\}|[^;{}]*;)", text):
        if re.search(r"\b(return|break)\b", m.group(2)):
            yield from re.findall(r"\bsz_mbar_wait\w*", m.group(1))


@pytest.mark.parametrize("name", FILES)
def test_a_warp_leaves_a_wait_as_a_whole(name):
    waits = list(leaving_waits(open(os.path.join(CSRC, name)).read()))
    assert waits and set(waits) == {"sz_mbar_wait_warp"}


def test_the_warps_wait_is_a_vote():
    text = open(os.path.join(CSRC, "sz_common.cuh")).read()
    assert re.search(r"bool sz_mbar_wait_warp\([^)]*\) \{ return __all_sync\(0xffffffffu, sz_mbar_wait\(bar, phase\)\); \}", text)
