"""What choosing a chunk length by the cost model (plan_core.cpp cheapestChunk)
adds to planning: the planner with it and without, in turn, on lists of long
requests (the best of several runs each, at most twice the time)."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
SRC = r'''
#include <chrono>
#include <string>
#include "%s/mtgp_gb300/csrc/plan_core.h"
using namespace mtgp;
extern "C" double seconds(const uint64_t *counts, int n, int sms, int reps) {
    std::vector<mtgp_work_item_t> it((size_t)n);
    uint64_t off = 0;
    for (int k = 0; k < n; k++) {
        it[k] = mtgp_work_item_t{};
        it[k].stream = (uint32_t)k;
        it[k].count = counts[k];
        it[k].out_offset = off;
        off += 4 * counts[k];
    }
    PlanOptions o;
    o.nstreams = n;
    o.can_jump = true;
    o.resident = 1520;
    o.sms = sms;
    PlanResult R;
    std::string err;
    double best = 1e9;
    for (int q = 0; q < reps; q++) {
        const auto t = std::chrono::steady_clock::now();
        if (planCore(it.data(), n, o, &R, &err)) return -1;
        best = std::min(best, std::chrono::duration<double>(
                                  std::chrono::steady_clock::now() - t).count());
    }
    return best;
}
'''


@pytest.mark.parametrize("n,median", [(4096, 65536), (10000, 65536), (100000, 65536)])
def test_planning_time(tmp_path, n, median):
    src, so = tmp_path / "p.cpp", tmp_path / "p.so"
    src.write_text("#include <algorithm>\n" + SRC % ROOT)
    subprocess.check_call(["g++", "-O3", "-std=c++17", "-shared", "-fPIC", "-o", str(so), str(src),
                           os.path.join(ROOT, "mtgp_gb300", "csrc", "plan_core.cpp")])
    f = ctypes.CDLL(str(so)).seconds
    f.restype = ctypes.c_double
    rng = np.random.default_rng(42)
    c = np.clip(np.rint(rng.lognormal(np.log(median), 1.0, n)), 1, 2 ** 22).astype(np.uint64)
    p = c.ctypes.data_as(ctypes.c_void_p)
    plain, model = 1e9, 1e9
    for _ in range(4):
        plain, model = min(plain, f(p, n, 0, 4)), min(model, f(p, n, 152, 4))
    assert 0 < plain and 0 < model < 2 * plain
