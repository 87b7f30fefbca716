"""A wait that runs out ends its warp as a whole: a lane that left a loop alone would leave the others at a __syncwarp for good.

Read from the sources, since no wait may be made to run out in earnest.
"""

import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "geometric_nn_ops_b200", "csrc")
ONE_LANE = re.compile(r"elect_one\(\)|lane == 0|leader")
VOTE = "__all_sync(0xffffffffu, "


def _blocks(text):
    """(header, body, headers around it) of every block in braces."""
    stack = []
    for m in re.finditer(r"[{}]", text):
        if m.group() == "{":
            start = max(text.rfind(c, 0, m.start()) for c in "{}") + 1
            stack.append((text[start:m.start()], m.end()))
        elif stack:
            header, begin = stack.pop()
            yield header, text[begin:m.start()], [h for h, _ in stack]


def _last_line(header):
    return header.rstrip().rpartition("\n")[2]


def _lone_exits(text):
    text = re.sub(r"//[^\n]*", "", text)
    blocks = list(_blocks(text))
    meets = {m.group(1) for h, body, _ in blocks if "__syncwarp()" in body and (m := re.search(r"auto (\w+) = \[", _last_line(h)))}
    for header, body, around in blocks:
        head = _last_line(header)
        if not re.search(r"\bfor \(", head) or any(ONE_LANE.search(_last_line(h)) for h in [*around, header]):
            continue
        if "__syncwarp()" not in body and not any(re.search(rf"\b{name}\(", body) for name in meets):
            continue
        waits = [line for line in body.split("\n") if "mbar_wait" in line and VOTE not in line]
        by_header = re.search(r"&& ok;", head) and any(re.search(r"\bok = ", line) for line in waits)
        by_break = re.search(r"if \(!mbar_wait[^\n]*break;", body) or re.search(r"ok = mbar_wait[^\n]*\n\s*if \(!ok\) break;", body)
        if by_header or by_break:
            yield head.strip()


@pytest.mark.parametrize("name", sorted(os.path.basename(f) for f in glob.glob(os.path.join(CSRC, "tc_*.cu*"))))
def test_no_lane_leaves_alone(name):
    with open(os.path.join(CSRC, name)) as f:
        assert list(_lone_exits(f.read())) == []
