"""Chunk lengths that go with the grid of all resident CTAs: equal runs that
fit it at once stay uncut, and of very many tasks the long ones are cut
shorter than the even share alone asks for.  On the host code over a fake CUDA
runtime of 152 SMs and 1520 resident CTAs."""
import ctypes

import numpy as np
import pytest

from mtgp_gb300.params import load_table


def plan(table, lens):
    """(tasks, chunk length; 0 = no run was cut)"""
    import fake_gpu
    from mtgp_gb300._lib import WorkItem
    fake = fake_gpu.load()
    L = fake.lib
    bits = int(table[4:6])
    fn = lambda name: getattr(L, "mtgp%d_gpu_%s" % (bits, name))  # noqa: E731
    p = load_table(table)[0]
    n = len(lens)
    seeds = np.zeros(n, dtype="u%d" % (bits // 8))
    idx = np.zeros(n, dtype=np.int32)
    pool, pl = ctypes.c_void_p(), ctypes.c_void_p()
    assert fn("pool_create")(ctypes.byref(pool), ctypes.byref(p), 1,
                             idx.ctypes.data_as(ctypes.c_void_p),
                             seeds.ctypes.data_as(ctypes.c_void_p), n) == 0
    it, off = (WorkItem * n)(), 0
    for k, c in enumerate(lens):
        it[k] = WorkItem(k, 0, int(c), off, 0)
        off += int(c) * (bits // 8)
    assert fn("pool_plan")(pool, it, n, ctypes.byref(pl)) == 0
    tasks, chunk = ctypes.c_int64(), ctypes.c_int64()
    assert L.mtgp_gpu_plan_info(pl, ctypes.byref(tasks), ctypes.byref(chunk)) == 0
    L.mtgp_gpu_plan_free(pl)
    fn("pool_free")(pool)
    return tasks.value, chunk.value


@pytest.mark.parametrize("table,n,log2", [("mtgp32_fast_23209", 400, 20),
                                          ("mtgp32_fast_11213", 640, 18),
                                          ("mtgp64dc_fast_11213", 640, 18)])
def test_equal_runs_of_one_round_of_all_are_not_cut(table, n, log2):
    assert plan(table, [1 << log2] * n) == (n, 0)


def test_long_runs_among_very_many():
    rng = np.random.default_rng(42)
    lens = np.clip(np.rint(rng.lognormal(np.log(16384), 1.0, 10000)), 1, 2 ** 22)
    tasks, chunk = plan("mtgp32_fast_11213", lens)
    assert tasks > 10000 and chunk < 393216
