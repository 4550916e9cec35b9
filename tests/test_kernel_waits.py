"""Bounded waits in code that a whole warp runs: no lane may branch on an answer of its own, or the lanes that go on wait for good
at the next vote, shuffle or tensor-memory instruction for those that left.  Read from the sources: no healthy run reaches it."""

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "uma_qmoe_b200" / "csrc"
DRAIN = re.compile(r"(^|\))\s*mbar_wait\([^;]*;")            # its answer is not used: copies in flight after a failure


@pytest.mark.parametrize("name", ["grouped.cu", "grouped_ts.cu", "grouped_wide.cu", "grouped_pair.cu"])
def test_no_lane_branches_on_its_own_wait(name):
    text = re.sub(r"//[^\n]*", "", (CSRC / name).read_text())
    if name == "grouped_pair.cu":                             # a single lane produces and issues there
        text = text[text.index("const int ct = tid - 256"):]
    for statement in re.split(r"(?<=[;{}])", text):
        if re.search(r"\bmbar_wait\(", statement):
            assert "__all_sync(" in statement or DRAIN.search(statement), statement
    assert "!*abort_flag" not in text                         # whether to go on with the next tile, likewise


def test_no_decode_lane_branches_on_its_own_wait():
    text = (CSRC / "decode.cu").read_text()
    wait = text[text.index("bool wait_or_fail("):]
    wait = wait[:wait.index("\n}\n")]
    assert wait.count("mbar_try_wait") == wait.count("__all_sync(0xffffffffu, mbar_try_wait") == 2
    assert "__any_sync(0xffffffffu, *fail ||" in wait and "!*fail" not in text
    body = text[text.index("decode_down_kernel("):]
    assert body.count("!s_fail") == 1                         # behind the CTA's barrier, where nobody sets it any more
