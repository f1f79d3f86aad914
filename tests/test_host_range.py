"""Which host arrays the state and force kernels may touch in place
(csrc/host_range.h): those that one page-locked range holds from the first
byte to the last.  Page-locked ranges are a table here, so that no kernel
meets a gap."""
import ctypes
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tooling_gb300", "csrc")
SOURCE = """
#include "host_range.h"
// ranges: host start, device start, bytes
extern "C" unsigned long long address(unsigned long long p, unsigned long long bytes, const unsigned long long* t, int n) {
  return device_address((const void*)p, bytes, [&](const void* q) {
    for (int k = 0; k < n; ++k)
      if ((uintptr_t)q >= t[3 * k] && (uintptr_t)q - t[3 * k] < t[3 * k + 2])
        return HostRange{(uintptr_t)q - t[3 * k] + t[3 * k + 1], t[3 * k + 1], t[3 * k + 2]};
    return HostRange{};
  });
}
"""


@pytest.fixture(scope="module")
def address(tmp_path_factory):
    d = tmp_path_factory.mktemp("host_range")
    (d / "t.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, str(d / "t.cpp"), "-o", str(d / "t.so")], check=True)
    f = ctypes.CDLL(str(d / "t.so")).address
    f.restype = ctypes.c_ulonglong
    f.argtypes = [ctypes.c_ulonglong, ctypes.c_ulonglong, ctypes.POINTER(ctypes.c_ulonglong), ctypes.c_int]

    def call(p, n, *ranges):
        flat = [x for r in ranges for x in r]
        return f(p, n, (ctypes.c_ulonglong * max(1, len(flat)))(*flat), len(ranges))
    return call


PAGE = 4096


@pytest.mark.parametrize("shift", [0, 1 << 40])  # the device's addresses equal the host's, or do not
def test_only_an_array_inside_one_range_is_used_in_place(address, shift):
    r = (16 * PAGE, 16 * PAGE + shift, 4 * PAGE)
    for p, n in ((16 * PAGE, 4 * PAGE), (16 * PAGE, 4), (17 * PAGE + 12, PAGE), (20 * PAGE - 4, 4)):
        assert address(p, n, r) == p + shift
    for p, n in ((16 * PAGE, 4 * PAGE + 4), (20 * PAGE - 4, 8), (16 * PAGE - 4, 8), (20 * PAGE, 4), (8 * PAGE, PAGE),
                 (17 * PAGE, 0), (17 * PAGE, 2 ** 64 - 1)):
        assert address(p, n, r) == 0
    assert address(17 * PAGE, 8) == 0


def test_two_ranges_with_memory_between_them_are_not_one(address):
    a, b = (16 * PAGE, 16 * PAGE, PAGE), (20 * PAGE, 20 * PAGE, PAGE)
    assert address(16 * PAGE + 64, 4 * PAGE + 64, a, b) == 0  # both ends page-locked, three pages between them not
    assert address(16 * PAGE, 5 * PAGE, a, b) == 0
    assert address(16 * PAGE, 2 * PAGE, a, (17 * PAGE, 17 * PAGE, PAGE)) == 0  # side by side, locked apart
