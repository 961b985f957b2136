"""How many splits a single-session launch of the tcgen05 decode kernels takes (csrc/split_bounds.h, compiled here as plain C++): against the same estimate over
every number of splits."""
import ctypes as C
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "miinfer_b200" / "csrc"
SOURCE = """
#include "split_bounds.h"
extern "C" uint32_t pick(uint32_t tiles, uint32_t most, uint32_t on_time, const uint32_t* c) {
    return b200kv::cheapest_splits(tiles, most, on_time, b200kv::SplitCosts{c[0], c[1], c[2], c[3], c[4], c[5]});
}
"""


@pytest.fixture(scope="module")
def native(tmp_path_factory):
    tmp = tmp_path_factory.mktemp("split_counts")
    (tmp / "shim.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", f"-I{CSRC}", str(tmp / "shim.cpp"), "-o", str(tmp / "shim.so")], check=True, capture_output=True)
    return C.CDLL(str(tmp / "shim.so"))


# splits that fit, splits that start on time, costs: 8, 4, 2 and 16 heads of 128, 4, 8 and 1 of 256, one split only
@pytest.mark.parametrize("most,on_time,costs", [(37, 33, (450, 900, 45, 0, 150, 5)), (74, 70, (450, 900, 45, 0, 150, 5)), (148, 144, (450, 900, 45, 0, 150, 5)),
                                                (18, 14, (450, 900, 45, 0, 150, 5)), (18, 0, (450, 900, 45, 0, 150, 5)), (37, 35, (850, 850, 70, 500, 0, 0xFFFFFFFF)),
                                                (18, 17, (850, 850, 70, 500, 0, 0xFFFFFFFF)), (148, 140, (850, 850, 70, 500, 0, 0xFFFFFFFF)), (1, 1, (850, 850, 70, 500, 0, 0xFFFFFFFF))])
def test_counts(native, most, on_time, costs):
    early, tile, split, late, per_late, fill = costs

    def cost(tiles, s):
        longest = -(-tiles // s)
        return min(longest, 3) * early + max(longest - 3, 0) * tile + s * split + (late + (s - on_time) * per_late if s > on_time else 0)

    c = (C.c_uint32 * 6)(*costs)
    for tiles in [*range(0, 400), 1023, 1024, 1025, 8191, 1 << 20]:
        got = native.pick(tiles, most, on_time, c)
        assert 1 <= got <= max(1, min(most, tiles)), (tiles, got)
        if tiles == 0 or most == 1:
            continue
        longest = -(-tiles // got)
        fewest = -(-tiles // longest)
        shortest = -(-tiles // most)
        best = min(cost(tiles, s) for s in range(1, min(most, tiles) + 1) if -(-tiles // s) <= shortest + 8)
        assert cost(tiles, fewest) == best, (tiles, got)
        if longest < fill:
            assert got == fewest, (tiles, got)
        else:   # no part is longer, and a launch whose splits all start on time stays one
            assert got >= fewest and (fewest > on_time or got <= on_time), (tiles, got)
