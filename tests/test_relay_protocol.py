"""What the relay kernel's hand-down between blocks rests on, read from its
source: a reader takes a strand for its group's by the tag beside it, so every
access to the hand-down row has to be one relaxed 8-byte word."""
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
