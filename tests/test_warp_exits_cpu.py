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


@pytest.mark.parametrize("name", ["decode_tc5.cu", "decode_tc5_wide.cu"])
def test_any_lane_poisons_its_partial(name):
    """These loops are not left: waits behind one that ran out are passed by, and the CTA's partial becomes NaN, whichever lane it was."""
    text = re.sub(r"//[^\n]*", "", (CSRC / name).read_text())
    at = [m.start() for m in re.finditer(r"atomicOr\(fail_flag", text)]
    assert len(at) == 1
    opened = []
    for i, c in enumerate(text[:at[0]]):
        if c == "{":
            opened.append(text[text.rfind("\n", 0, i) + 1:i])
        elif c == "}":
            opened.pop()
    guards = [g for g in opened + [text[text.rfind("\n", 0, at[0]) + 1:at[0]]] if re.search(r"\b(lane|tid)\b", g)]
    assert not guards, guards
