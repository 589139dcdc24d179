"""The closure kernel's groups share a block number in shared memory: the
leader writes it, the group's other warps read it.  On every way round the
block loop a group barrier has to lie between the write and the reads, and
between the reads and the next write; the order is read from the source."""
import os
import re

import pytest

SRC = os.path.join(os.path.dirname(__file__), "..", "rift_gb300", "csrc", "rift_closure.cu")


def _ways_round():
    """Events of one pass of k_closure's block loop, for a dry block (which ends
    at `continue`) and for a wet one: W writes T.next, R reads it, B barrier."""
    src = re.sub(r"//[^\n]*", "", open(SRC).read())
    body = src[src.index("void __launch_bounds__(TCT, 1) k_closure("):]
    body = body[body.index("for (; tile < ntile; tile = next)"):body.index("tcEnd(")]
    marks = r"(?P<W>T\.next = )|(?P<R>= T\.next;)|(?P<B>group(?:And|Sync)\()|(?P<D>if \(dry\) \{)|(?P<C>\n            continue;)"
    dry, wet, inside = [], [], False
    for m in re.finditer(marks, body):
        e = m.lastgroup
        if e == "D":
            inside = True
        elif e == "C":
            if inside:
                break
        else:
            dry.append(e)
            if not inside:
                wet.append(e)
    for m in re.finditer(marks, body[m.end():]):
        if m.lastgroup in "WRB":
            wet.append(m.lastgroup)
    return {"dry": dry, "wet": wet}


@pytest.mark.parametrize("first", ["dry", "wet"])
@pytest.mark.parametrize("second", ["dry", "wet"])
def test_block_number_is_ordered_by_barriers(first, second):
    ways = _ways_round()
    seq = [e for e in ways[first] + ways[second]]
    assert seq.count("W") == 2 and seq.count("R") == 2 and "B" in seq, seq
    last = None
    for e in seq:
        if e == "B":
            last = None
        else:
            assert last is None or last == e, (first, second, seq)
            last = e
