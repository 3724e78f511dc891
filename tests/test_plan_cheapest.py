"""The automatic chunk length of plans whose jumps are made ahead of the
launch (plan_core.cpp cheapestChunk), through the CPU probe's planner: every
value of every item is still produced once and in order for any number of SMs
(the driver of the check is test_plan_host's model), and nothing is cut where
no run is longer than the shortest jumped skip."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = r'''
#include <string>
#include "%s/mtgp_gb300/csrc/plan_core.h"
using namespace mtgp;
// out: chunk, tasks, total values, tasks that start at a jump; -1 on error,
// -2 when the pieces of a stream do not follow one another
extern "C" int cheapest(const uint64_t *counts, int n, int sms, int64_t *out) {
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
    o.sms = sms;
    PlanResult R;
    std::string err;
    if (planCore(it.data(), n, o, &R, &err)) return -1;
    std::vector<std::vector<const PlanTask *>> by((size_t)n);
    for (const PlanTask &t : R.tasks) by[t.stream].push_back(&t);
    out[0] = R.chunk;
    out[1] = (int64_t)R.tasks.size();
    out[2] = out[3] = 0;
    for (int k = 0; k < n; k++) {
        uint64_t done = 0;
        while (done < counts[k]) {
            const PlanTask *next = nullptr;
            for (const PlanTask *t : by[k])
                if (t->run + t->off == done && t->total) next = t;
            if (!next) return -2;
            done += next->total;
            out[3] += next->off != 0;
        }
        if (done != counts[k]) return -2;
        out[2] += (int64_t)done;
    }
    return 0;
}
'''


@pytest.fixture(scope="module")
def cheapest(tmp_path_factory):
    root = os.path.dirname(HERE)
    d = tmp_path_factory.mktemp("cheapest")
    src, so = d / "p.cpp", d / "p.so"
    src.write_text(SRC % root)
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-o", str(so), str(src),
                           os.path.join(root, "mtgp_gb300", "csrc", "plan_core.cpp")])
    f = ctypes.CDLL(str(so)).cheapest

    def run(counts, sms):
        c = np.asarray(counts, dtype=np.uint64)
        out = np.zeros(4, dtype=np.int64)
        rc = f(c.ctypes.data_as(ctypes.c_void_p), len(c), sms, out.ctypes.data_as(ctypes.c_void_p))
        assert rc == 0
        return [int(v) for v in out]
    return run


def test_short_runs_are_not_cut(cheapest):
    assert cheapest([1 << 17] * 1000, 152) == [0, 1000, 1000 << 17, 0]
    assert cheapest([1], 152) == [0, 1, 1, 0]


@pytest.mark.parametrize("sms", [1, 7, 152])
@pytest.mark.parametrize("n,median", [(1, 1 << 30), (3, 200000), (50, 60000), (2000, 65536)])
def test_every_value_once(cheapest, n, median, sms):
    rng = np.random.default_rng(n)
    counts = np.clip(np.rint(rng.lognormal(np.log(median), 1.0, n)), 1, 2 ** 33).astype(np.int64)
    counts[0] = max(int(counts[0]), (1 << 17) + 1)
    chunk, tasks, total, jumps = cheapest(counts, sms)
    assert total == counts.sum() and tasks == n + jumps


def test_equal_runs_fill_the_slots(cheapest):
    # 200 runs of 2^20 on 608 slots: three pieces each, one round
    chunk, tasks, _, _ = cheapest([1 << 20] * 200, 152)
    assert tasks == 600
