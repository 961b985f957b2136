"""The reference maximum that suffix attention hands from tile to tile (csrc/reference_word.h, compiled here as plain C++): a thread goes on with the value it has published,
whatever the threads of later tiles have put into the word by the time it reads it back."""
import ctypes as C
import re
import struct
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "miinfer_b200" / "csrc"
SOURCE = """
#include "reference_word.h"
extern "C" unsigned long long word(uint32_t value, uint32_t seq) { return b200kv::reference_word(value, seq); }
extern "C" uint32_t own(uint32_t found, uint32_t mine) { return b200kv::own_reference(found, mine); }
"""


@pytest.fixture(scope="module")
def native(tmp_path_factory):
    tmp = tmp_path_factory.mktemp("reference_word")
    (tmp / "shim.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", f"-I{CSRC}", str(tmp / "shim.cpp"), "-o", str(tmp / "shim.so")], check=True, capture_output=True)
    lib = C.CDLL(str(tmp / "shim.so"))
    lib.word.restype, lib.word.argtypes = C.c_ulonglong, [C.c_uint32, C.c_uint32]
    lib.own.restype, lib.own.argtypes = C.c_uint32, [C.c_uint32, C.c_uint32]
    return lib


def bits(x):
    return struct.unpack("I", struct.pack("f", x))[0]


@pytest.mark.parametrize("values", [(-3.0, 6.0, 15.5, 24.0), (float("-inf"), float("-inf"), 0.0, 9.0), (0.0, 0.0, 0.0, 0.0), (float("nan"), 1.0, 10.0, 19.0)])
def test_own_value_whatever_the_word_holds(native, values):
    """Tile t publishes, up to three later tiles overwrite the word before it is read back: the outcome is what tile t published, and what rescales the row's output."""
    for first in (0, 1, 7, (1 << 31) - 5):      # tiles of 64 of at most 2^32 positions: far fewer
        for t, v in enumerate(values):
            for later in range(t, len(values)):     # the last tile to have published by then
                found = native.word(bits(values[later]), first + later + 1)
                assert found & 0xFFFFFFFF == bits(values[later])
                assert native.own(found >> 32, bits(v)) == bits(v)


def test_no_value_is_taken_from_the_word_behind_the_store():
    """In the softmax loop only the number above the value is read back, and goes through that function alone."""
    text = re.sub(r"//[^\n]*", "", (CSRC / "prefill_tc5.cu").read_text())
    reads = re.findall(r'asm volatile\("ld\.volatile\.shared\.(\w+) %0[^;]*;" : "=\w"\((\w+)\) : "r"\(([^;]*)\) : "memory"\);', text)
    assert len(reads) == len(re.findall(r"ld\.volatile\.shared", text)) == 1
    width, name, address = reads[0]
    assert width == "u32" and address.endswith(" + 4")
    uses = [line for line in text.splitlines() if re.search(rf"\b{name}\b", line) and "asm volatile" not in line and f" {name};" not in line]
    assert len(uses) == 1 and f"own_reference({name}, " in uses[0]
