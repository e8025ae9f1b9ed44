"""CPU: no kernel holds a warp-wide instruction in inline assembly that the compiler may move. A plain asm
statement is a pure function of its operands to the compiler, which may sink it into a branch that only some
lanes take; an instruction for a full mask of lanes is then undefined. Only volatile asm stays in place."""

import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ssdf_b200", "csrc")


def test_no_movable_warp_instruction():
    movable = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))
                       + glob.glob(os.path.join(CSRC, "*.h"))):
        with open(path) as f:
            text = f.read()
        for m in re.finditer(r"\basm(\s+volatile)?\s*\(", text):
            body = text[m.end():text.index(";", text.index(")", m.end()))]
            if not m.group(1) and re.search(r"\b(redux|shfl|vote|match|bar|barrier)\.", body):
                movable.append((os.path.basename(path), body.strip()[:60]))
    assert not movable, movable
