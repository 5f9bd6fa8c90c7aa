"""The pair walk copies a target's row places to shared memory asynchronously
while its first candidates are evaluated.  Whoever reads them has to wait for
the copy first: a row read too early is the warp's previous row, or at a warp's
first target whatever the shared memory held, and a count is then written
there.  Whether the copy has arrived is a matter of time, so no run shows a
missing wait reliably; the source does."""

import os
import re

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "yggdrax_b200",
                   "csrc", "pair_walk.cuh")


def _functions():
    """(name, body) of every device function, comments removed."""
    text = re.sub(r"//[^\n]*", "", open(SRC).read())
    out = {}
    for m in re.finditer(r"\b(pw_\w+|k_\w+)\(", text):
        depth, i = 0, m.end() - 1
        while True:
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
            if depth == 0:
                break
        rest = text[i:].lstrip()
        if not rest.startswith("{"):
            continue  # a call
        start = j = text.index("{", i)
        depth = 0
        while True:
            depth += {"{": 1, "}": -1}.get(text[j], 0)
            j += 1
            if depth == 0:
                break
        out[m.group(1)] = text[start:j]
    return out


def test_every_reader_of_a_row_waits_for_its_copy():
    readers = {k: b for k, b in _functions().items() if "W.row[" in b.replace("&W.row[", "")}
    assert {"pw_flush_row", "pw_hand_off", "k_pair_walk"} <= set(readers)
    for name, body in readers.items():
        if name == "k_pair_walk":
            continue
        assert -1 < body.find("pw_copy_wait()") < body.find("W.row["), name
    # the walk itself reads a row after its piece, whose end waits whatever
    # the piece did: outside of every loop and condition
    walk = readers["k_pair_walk"]
    read = walk.replace("&W.row[", "&______").index("W.row[")
    assert walk.index("pw_copy16(") < walk.index("pw_run_piece<") < read
    piece = _functions()["pw_run_piece"]
    waits = [m.start() for m in re.finditer(r"pw_copy_wait\(\)", piece)]
    assert any(piece[:w].count("{") - piece[:w].count("}") == 1 for w in waits)
