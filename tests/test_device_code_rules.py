"""Rules of the device code that no run can be relied on to show when they are
broken, checked on the source: on one warp and one GPU the broken form usually
gives the right result."""

from __future__ import annotations

import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "cujpegxl_b200" / "csrc"


def _loops(text: str):
    """Bodies of the for loops of `text` that hold no other loop."""
    for m in re.finditer(r"\bfor \([^\n]*\) \{", text):
        depth, at = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[at], 0)
            at += 1
        body = text[m.end():at]
        if "for (" not in body:
            yield body


def test_rounds_of_shared_counters_are_ordered():
    """A loop whose lanes take turns at a shared counter by __match_any_sync
    (the leader of a group may be another lane in the next round) adds
    atomically or ends its rounds with a warp barrier: the match alone does not
    order memory."""
    turns = [b for b in _loops((CSRC / "entropy.cu").read_text())
             if "__match_any_sync" in b and re.search(r"\b\w+\.\w+\[\w+\] \+= ", b)]
    assert len(turns) >= 3
    for body in turns:
        assert body.rstrip().rstrip("}").rstrip().endswith("__syncwarp();"), body


def test_chained_passes_read_by_ordinary_loads():
    """A kernel launched on programmatic stream serialisation can be resident
    while the grid before it still writes, so what that grid writes is not
    read-only for the kernel's lifetime: no read-only-cache loads."""
    for name in ("entropy.cu", "cujpegxl.cu"):
        text = (CSRC / name).read_text()
        assert "launch_chained(" in text
        assert "__ldg(" not in text and "ld.global.nc" not in text and "__restrict__" not in text, name
