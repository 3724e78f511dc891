"""How many CTAs a plan's launch asks for (0: all that fit): few per SM only
where the longest tasks set the launch's length.  On the host code over a fake CUDA
runtime of 152 SMs."""
import ctypes

import numpy as np
import pytest

from mtgp_gb300.params import load_table


def grid(table, lens, core=2, kinds=None):
    import fake_gpu
    from mtgp_gb300._lib import WorkItem
    fake = fake_gpu.load()
    L = fake.lib
    bits = int(table[4:6])
    fn = lambda name: getattr(L, "mtgp%d_gpu_%s" % (bits, name))  # noqa: E731
    fake.clear()
    p = load_table(table)[0]
    n = len(lens)
    seeds = np.zeros(n, dtype="u%d" % (bits // 8))
    idx = np.zeros(n, dtype=np.int32)
    pool, plan = ctypes.c_void_p(), ctypes.c_void_p()
    assert fn("pool_create")(ctypes.byref(pool), ctypes.byref(p), 1,
                             idx.ctypes.data_as(ctypes.c_void_p),
                             seeds.ctypes.data_as(ctypes.c_void_p), n) == 0
    assert fn("pool_set_tuning")(pool, b"core", core) == 0
    it, off = (WorkItem * n)(), 0
    for k, c in enumerate(lens):
        it[k] = WorkItem(k, 0 if kinds is None else kinds[k], int(c), off, 0)
        off += int(c) * (bits // 8)
    assert fn("pool_plan")(pool, it, n, ctypes.byref(plan)) == 0
    fake.clear()
    assert L.mtgp_gpu_plan_launch(plan, ctypes.create_string_buffer(1), None) == 0
    got = [l for l in fake.log() if l.startswith("launchBatch")]
    L.mtgp_gpu_plan_free(plan)
    fn("pool_free")(pool)
    assert len(got) == 1
    return int(got[0].split()[2])


CASES = [("mtgp32_fast_11213", 608), ("mtgp64dc_fast_11213", 608), ("mtgp32_fast_23209", 304)]


@pytest.mark.parametrize("table,few", CASES)
def test_short_or_equal_tasks_take_every_slot(table, few):
    assert grid(table, [1000] * 4000) == 0
    assert grid(table, [1 << 17] * (few + 1)) == 0  # two rounds on few
    assert grid(table, [1 << 14] * 700, kinds=[0, 1] * 350) == 0


@pytest.mark.parametrize("table,few", CASES)
def test_long_tasks_take_few(table, few):
    assert grid(table, [1 << 17] * few) == few
    assert grid(table, [1 << 17] + [1000] * 3 * few) == few
    # so many short requests that the work as a whole sets the length
    assert grid(table, [1 << 17] + [1000] * 9 * few) == 0


def test_four_word_core_takes_every_slot():
    assert grid("mtgp32_fast_11213", [1 << 17] * 100, core=4) == 0
