"""CPU check of the grouped M2L's limits (csrc/m2l_size.h): rows are numbered by
32-bit integers in units of eight entries, and the memory of rows, tensors and
operators decides whether a call that can go pair by pair takes the products."""
import ctypes
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fmm_gb300", "csrc")
SOURCE = """
#include "m2l_size.h"
extern "C" int fit(long long units) { return fmm::m2l_rows_fit(units); }
extern "C" double bytes(long long pairs, long long groups, int row, int tensor, long long op, int entry) {
    return fmm::m2l_bytes({pairs, groups, row, tensor, op, entry});
}
extern "C" double limit() { return fmm::kGroupedBytes; }
extern "C" int unit() { return fmm::kRowUnit; }
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("m2l_size")
    src, so = d / "t.cpp", d / "t.so"
    src.write_text(SOURCE)
    subprocess.check_call(["g++", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, "-o", str(so), str(src)])
    lib = ctypes.CDLL(str(so))
    lib.fit.argtypes = [ctypes.c_longlong]
    lib.bytes.restype = lib.limit.restype = ctypes.c_double
    lib.bytes.argtypes = [ctypes.c_longlong, ctypes.c_longlong, ctypes.c_int, ctypes.c_int, ctypes.c_longlong,
                          ctypes.c_int]
    return lib


def row(p, full=False):
    k = (p + 1) * (p + 2) * (p + 3) // 6 if full else (p + 1) ** 2
    return -(-k // 8) * 8


@pytest.mark.parametrize("p,pairs", [(5, 429_496_729), (4, 536_870_911), (10, 134_217_727), (12, 97_612_893)])
def test_row_numbers(lib, p, pairs):
    """The last row's number is the first one past 2^31 - 1 just above `pairs`."""
    units = row(p) // lib.unit()
    assert lib.fit(units * pairs)
    assert not lib.fit(units * (pairs + 1))
    assert not lib.fit(units * 4 * pairs)  # where 32 bits come round to positive numbers again


def test_memory(lib):
    # default call of 20 million particles: 4e8 pairs, order 5: rows alone are 128 GB
    assert lib.bytes(400_000_000, 300_000, row(5), 121, 0, 8) > 128e9 > lib.limit()
    # 5e6 groups of two pairs at order 12 over all components: the tensors, not the rows
    rows = 1e7 * row(12, True) * 8
    assert rows < lib.limit() < lib.bytes(10_000_000, 5_000_000, row(12, True), 2925, 0, 8)
    # operators of many groups: no more than a batch
    few = lib.bytes(1000, 10, 40, 121, 1 << 18, 8)
    assert few == pytest.approx(1000 * (320 + 44) + 10 * 121 * 8 + 10 * (1 << 18))
    assert lib.bytes(10_000_000, 1_000_000, 40, 121, 1 << 18, 8) < 10_000_000 * 364 + 1e6 * 968 + 16.1e9
    # what calls take in earnest stays: a million particles at order 5, 60,000 at order 10
    assert lib.bytes(20_000_000, 10_000, row(5), 121, 1 << 18, 8) < lib.limit()
    assert lib.bytes(3_000_000, 20_000, row(10), 441, 1 << 18, 8) < lib.limit()
