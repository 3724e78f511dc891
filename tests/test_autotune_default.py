"""The autotuner measures what the pool would do by itself: the plan that
pool_plan makes is among its candidates, the automatic grid also for its own
chunk lengths.  On the host code over a fake CUDA runtime, whose launches all
take the same time (the first candidate is kept)."""
import ctypes

import numpy as np
import pytest

from mtgp_gb300.params import load_table


@pytest.mark.parametrize("table", ["mtgp32_fast_11213", "mtgp64dc_fast_11213"])
def test_default_plan_is_a_candidate(table):
    import fake_gpu
    from mtgp_gb300._lib import WorkItem
    fake = fake_gpu.load()
    L = fake.lib
    bits = int(table[4:6])
    fn = lambda name: getattr(L, "mtgp%d_gpu_%s" % (bits, name))  # noqa: E731
    p, n = load_table(table)[0], 300
    rng = np.random.default_rng(42)
    lens = np.clip(np.rint(rng.lognormal(np.log(65536), 1.0, n)), 1, 2 ** 22).astype(np.int64)
    seeds, idx = np.zeros(n, dtype="u%d" % (bits // 8)), np.zeros(n, dtype=np.int32)
    pool, plain, best = ctypes.c_void_p(), ctypes.c_void_p(), ctypes.c_void_p()
    fake.clear()
    assert fn("pool_create")(ctypes.byref(pool), ctypes.byref(p), 1,
                             idx.ctypes.data_as(ctypes.c_void_p),
                             seeds.ctypes.data_as(ctypes.c_void_p), n) == 0
    it, off = (WorkItem * n)(), 0
    for k, c in enumerate(lens):
        it[k] = WorkItem(k, 0, int(c), off, 0)
        off += int(c) * (bits // 8)
    out = ctypes.create_string_buffer(1)

    def launch(plan):
        fake.clear()
        assert L.mtgp_gpu_plan_launch(plan, out, None) == 0
        return [l for l in fake.log() if l.startswith("launchBatch")]

    assert fn("pool_plan")(pool, it, n, ctypes.byref(plain)) == 0
    want = launch(plain)
    report = ctypes.create_string_buffer(1 << 16)
    fake.clear()
    assert fn("pool_autotune")(pool, it, n, out, None, 1, ctypes.byref(best), report, 1 << 16) == 0
    tried = [l for l in fake.log() if l.startswith("launchBatch")]
    assert want[0] in tried
    assert "grid 608" in want[0]  # an uneven list: few CTAs per SM
    assert len({l for l in tried if "grid 608 " in l}) > 3  # with other lengths too
    assert launch(best) == want
    assert b"grid=auto" in report.value and b"608 CTAs" in report.value
    L.mtgp_gpu_plan_free(plain)
    L.mtgp_gpu_plan_free(best)
    fn("pool_free")(pool)
