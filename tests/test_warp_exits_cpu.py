"""Loops of the device code that hold warp-wide instructions (aligned TMEM accesses, MMAs, votes, shuffles) are left by whole warps: a bounded wait that runs out for
single lanes would otherwise leave the others with an instruction that waits for them.  Such a wait cannot be made to run out here, so the source is read."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "miinfer_b200" / "csrc"


def bodies(text, head):
    """The bodies of the loops that begin with `head`."""
    found = []
    for m in re.finditer(re.escape(head), text):
        start = text.index("{", m.end() - 1)
        depth = 0
        for end in range(start, len(text)):
            depth += {"{": 1, "}": -1}.get(text[end], 0)
            if depth == 0:
                found.append(text[start:end])
                break
    return found


@pytest.mark.parametrize("name,head", [("prefill_tc5.cu", "for (int j = grp; j < nt; j += 2) {"), ("decode_q8.cu", "for (int i = 0; i < ntiles; ++i) {")])
def test_left_by_whole_warps(name, head):
    loops = bodies(re.sub(r"//[^\n]*", "", (CSRC / name).read_text()), head)
    assert len(loops) == 1 and re.search(r"_sync\(|tmem_ld|mma_", loops[0])
    exits = [line for line in loops[0].splitlines() if re.search(r"\b(break|return|continue|goto)\b", line)]
    assert exits
    for line in exits:
        assert re.search(r"if \(!?(__any_sync|__all_sync|mbar_wait_warp)\(", line), line.strip()
