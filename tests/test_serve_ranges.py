"""The look-up of a batch's destinations in device memory (server_core.h
RangeMap): the range that holds an address and what is left of it, and no time
that grows with the number of ranges (a batch may have as many allocations as
requests)."""
import ctypes
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = r'''
#include <algorithm>
#include <chrono>
#include "%s/mtgp_gb300/csrc/server_core.h"
using namespace mtgp;
extern "C" int check() {
    RangeMap m;
    if (m.left(0) || m.left(1000) || m.left(~0ULL)) return 1;
    m.add(4096, 512);
    m.add(0x7f0000000000, 1 << 20);
    m.add(4608, 64);  // right behind the first
    const uint64_t at[][2] = {{4095, 0}, {4096, 512}, {4607, 1}, {4608, 64}, {4671, 1}, {4672, 0},
                              {4096, 512}, {0x7f0000000000, 1 << 20}, {0x7f00000fffff, 1},
                              {0x7f0000100000, 0}, {0, 0}, {4700, 0}, {~0ULL, 0}};
    for (auto &a : at)
        if (m.left(a[0]) != a[1]) return 2;
    return 0;
}
// seconds for n ranges, each added when it is first asked for and asked twice
extern "C" double seconds(int n) {
    RangeMap m;
    const auto t = std::chrono::steady_clock::now();
    for (int q = 0; q < 2; q++)
        for (uint64_t k = 0; k < (uint64_t)n; k++) {
            const uint64_t a = 4096 * (1 + (k * 7919) %% (uint64_t)n);
            if (!m.left(a)) m.add(a, 256);
            if (m.left(a) != 256) return -1;
        }
    return std::chrono::duration<double>(std::chrono::steady_clock::now() - t).count();
}
'''


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("ranges")
    src, so = d / "p.cpp", d / "p.so"
    src.write_text(SRC % ROOT)
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-o", str(so), str(src)])
    return ctypes.CDLL(str(so))


def test_ranges(lib):
    assert lib.check() == 0


def test_many_ranges(lib):
    lib.seconds.restype = ctypes.c_double
    assert 0 < lib.seconds(200000) < 5  # a search through a list takes minutes
