"""What the relay kernel's hand-down between blocks rests on, read from its
source: a reader takes a strand for its group's by the tag beside it, so every
access to the hand-down row has to be one relaxed 8-byte word; and a wait ends
for all lanes of a warp at once, with its status raised."""
import os
import re

import slcs

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(slcs.__file__))), "csrc", "relay.cu")


def _code():
    with open(SOURCE) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def test_row_words_are_moved_whole():
    code = _code()
    for op, name in (("ld", "ld_relaxed_pair"), ("st", "st_relaxed_pair")):
        body = re.search(r"%s\(.*?\n}" % name, code, re.S).group(0)
        assert re.search(r'"%s\.relaxed\.gpu\.global\.u64 ' % op, body)
    # The row pointer is made once and goes nowhere but into those two.
    uses = re.findall(r"[^\n]*\brow\b[^\n]*", code[code.index("relay_kernel("):])
    assert len(uses) >= 4
    made, rest = uses[0], uses[1:]
    assert "int2 *row = L.rows" in made and code.count("L.rows") == 1
    for line in rest:
        assert not re.sub(r"\b(ld|st)_relaxed_pair\(row \+ c\b", "", line).count("row"), line


def test_one_lane_ends_a_wait():
    """No vote over the lanes' own clocks: the limit is read, the status raised
    and the abort flag set under one lane's condition, whose answer all take."""
    code = _code()
    body = re.search(r"auto give_up = .*?\n            };", code, re.S).group(0)
    assert "__any_sync" not in body
    lane0 = body[body.index("if (lane == 0) {"):body.rindex("return")]
    for part in ("globaltimer_ns()", "raise_status(", "st_relaxed_gpu(", "L.wait_ns"):
        assert body.count(part) == lane0.count(part) == 1
    assert re.search(r"return __shfl_sync\(FULL_MASK, int\(over\), 0\) != 0;", body)
