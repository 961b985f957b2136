"""How a single-session launch of the streaming decode kernel divides its tiles among its splits (csrc/split_bounds.h, compiled here as plain C++)."""
import ctypes as C
import random
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "miinfer_b200" / "csrc"
SOURCE = """
#include "split_bounds.h"
extern "C" void bounds(uint32_t tiles, uint32_t splits, uint32_t late, uint32_t* out) {
    for (uint32_t i = 0; i < splits; ++i) {
        const b200kv::TileRange r = b200kv::split_tiles<8>(tiles, i, splits, late);
        out[2 * i] = r.begin, out[2 * i + 1] = r.end;
    }
}
extern "C" uint32_t late(int overlap, int inside, uint32_t heads, uint32_t splits, uint32_t mergers, uint32_t sms) {
    return b200kv::late_splits(overlap != 0, inside != 0, heads, splits, mergers, sms);
}
"""
WARPS, TILE = 8, 16
HYBRID, DENSE = (37, 12), (18, 4)     # splits and late ones on 148 SMs: 24 / 4 heads of 256, 32 / 8 heads of 128


@pytest.fixture(scope="module")
def native(tmp_path_factory):
    tmp = tmp_path_factory.mktemp("split_bounds")
    (tmp / "shim.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", f"-I{CSRC}", str(tmp / "shim.cpp"), "-o", str(tmp / "shim.so")], check=True, capture_output=True)
    return C.CDLL(str(tmp / "shim.so"))


def parts(native, tiles, splits, late):
    out = (C.c_uint32 * (2 * splits))()
    native.bounds(tiles, splits, late, out)
    begins, ends = out[::2], out[1::2]
    assert begins[0] == 0 and ends[-1] == tiles and begins[1:] == ends[:-1] and all(x <= y for x, y in zip(begins, ends))   # every tile once, in order
    return [y - x for x, y in zip(begins, ends)]


def rounds(tiles):
    return -(-tiles // WARPS)


@pytest.mark.parametrize("splits,late", [HYBRID, DENSE, (9, 4), (128, 63), (3, 1), (74, 8), (18, 8)])
def test_no_split_gets_another_round(native, splits, late):
    """Uneven parts: the longest has as many rounds as the longest even one (so a warp never has more tiles than the choice of the kernel assumes), the
    late ones one less, none is empty; and everywhere else the parts are even."""
    rng, seen = random.Random(splits), 0
    for tiles in [*range(0, 9 * splits * WARPS // 2), *(rng.randrange(1 << 28) for _ in range(2000)), (1 << 28) - 1]:
        even = parts(native, tiles, splits, 0)
        assert even == [tiles * (i + 1) // splits - tiles * i // splits for i in range(splits)]
        got = parts(native, tiles, splits, late)
        if got == even:
            continue
        seen += 1
        assert rounds(max(got)) == rounds(max(even)) >= 3
        assert rounds(max(got[-late:])) < rounds(max(even)) and min(got) > 0
        assert max(got[:-late]) - min(got[:-late]) <= 1 and max(got[-late:]) - min(got[-late:]) <= 1
    assert seen > 0


# lengths at which a split shorter by a round would cost the others one, and lengths at which it does not
@pytest.mark.parametrize("shape,even,uneven", [(HYBRID, (8000, 9105, 9200, 9472, 12673, 13500, 14208), (9500, 12000, 12672, 14209, 15000, 30000)),
                                               (DENSE, (4096, 4608, 6417, 6600, 6912, 8721, 9000, 9216, 11300, 13500), (4609, 5000, 6400, 7500, 8700, 10000, 12000, 30000))])
def test_lengths_that_keep_even_splits(native, shape, even, uneven):
    splits, late = shape
    for length in even + uneven:
        tiles = -(-length // TILE)
        assert (parts(native, tiles, splits, late) == parts(native, tiles, splits, 0)) == (length in even), length


def test_splits_start_late_only_behind_mergers_on_a_full_device(native):
    late = native.late
    assert late(1, 1, 4, 37, 12, 148) == 12 and late(1, 1, 8, 18, 4, 148) == 4      # the library's own split counts
    for heads, splits, mergers in ((4, 37, 12), (8, 18, 4)):
        assert late(0, 1, heads, splits, mergers, 148) == 0       # without launch overlap all CTAs start together
        assert late(1, 0, heads, splits, mergers, 148) == 0       # the merge is a kernel of its own
    assert late(1, 1, 8, 9, 4, 148) == 0 and late(1, 1, 1, 128, 1, 148) == 0        # there is room beside the mergers
    assert late(1, 1, 4, 37, 12, 147) == 13 and late(1, 1, 8, 18, 4, 176) == 0
    assert late(1, 1, 16, 9, 16, 148) == 0                        # most splits would be late ones
