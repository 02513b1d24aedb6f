"""Row-wise fetches of encoded weights stay inside the tensor (csrc/row_copy.h, compiled for the host; no GPU)."""
import ctypes
import os
import subprocess

import pytest

ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))

PROGRAM = r"""
#include "row_copy.h"
// Every box of every row of an [n][row_bytes] tensor: the number of boxes whose copy leaves the tensor, is not made of whole granules,
// overruns its slot or misses a byte.
extern "C" long long faults(unsigned long long row_bytes, unsigned long long n, unsigned long long span, unsigned long long pitch) {
    long long bad = 0;
    const unsigned long long total = row_bytes * n;
    for (unsigned long long row = 0; row < n; ++row) {
        for (unsigned long long from = row * row_bytes; from < (row + 1) * row_bytes; from += span) {
            unsigned long long to = from + span;
            if (to > (row + 1) * row_bytes) to = (row + 1) * row_bytes;
            const ribn::RowCopy c = ribn::row_copy(from, to, total);
            const bool inside = c.first + c.bytes <= total && c.first + c.bytes + c.tail <= total;
            const bool whole = c.first % 16 == 0 && c.bytes % 16 == 0 && c.tail % 2 == 0 && c.tail < 16;
            const bool covers = c.first <= from && c.first + c.bytes + c.tail >= to;
            const bool fits = c.bytes + c.tail <= pitch;
            // rows of all tiles (of 16) but the last are copied up to the next boundary without a look at the tensor's end
            const bool plain = row >= (n - 1) / 16 * 16 || (c.tail == 0 && c.first + c.bytes == ((to + 15) & ~15ull));
            if (!(inside && whole && covers && fits && plain)) ++bad;
        }
    }
    return bad;
}
"""


@pytest.fixture(scope="module")
def faults(tmp_path_factory):
    folder = tmp_path_factory.mktemp("row_copy")
    source, library = folder / "t.cpp", folder / "t.so"
    source.write_text(PROGRAM)
    subprocess.run([os.environ.get("CXX", "g++"), "-std=c++17", "-Wall", "-Werror", "-O1", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, "engine_b200", "csrc"), str(source), "-o", str(library)], check=True)
    function = ctypes.CDLL(str(library)).faults
    function.argtypes, function.restype = [ctypes.c_ulonglong] * 4, ctypes.c_longlong
    return function


# box span and slot pitch of the narrow kernel's row-wise fetches: eight super-blocks of Q6_K, thirty-two blocks of Q8_0
@pytest.mark.parametrize("block,span,pitch,counts", [(210, 1680, 1712, (1, 2, 3, 5, 8, 10, 20, 21, 43, 100)),
                                                     (34, 1088, 1104, (1, 2, 3, 7, 31, 32, 33, 127, 128, 129, 259))])
def test_copies_stay_inside_the_tensor(faults, block, span, pitch, counts):
    for per_row in counts:
        for n in (1, 2, 3, 7, 8, 15, 16, 17, 129, 5003):
            assert faults(block * per_row, n, span, pitch) == 0, (per_row, n)
