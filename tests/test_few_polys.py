"""Up to eight jump polynomials: one launch of a chain each where a cluster of
CTAs shares a product, a tree of products in three launches where one CTA works
alone (MEXP 110503, whose wide table does not fit in shared memory) and a
chain's seven products in turn would take twice as long.  On the host code over
a fake CUDA runtime, and on the GPU against the reference's PowerXMod
(mtgp-calc-jump.hpp:135-162, by way of the jumped windows)."""
import ctypes

import numpy as np
import pytest

from mtgp_gb300.params import load_table

STEPS = 0x123456789abcdef


@pytest.mark.parametrize("table,launches", [("mtgp64dc_fast_11213", 1), ("mtgp64_fast_44497", 1),
                                            ("mtgp64_fast_110503", 3)])
def test_launches(table, launches):
    import fake_gpu
    fake = fake_gpu.load()
    L = fake.lib
    fake.clear()
    p = load_table(table)[0]
    seeds, idx = np.zeros(1, dtype=np.uint64), np.zeros(1, dtype=np.int32)
    pool = ctypes.c_void_p()
    assert L.mtgp64_gpu_pool_create(ctypes.byref(pool), ctypes.byref(p), 1,
                                    idx.ctypes.data_as(ctypes.c_void_p),
                                    seeds.ctypes.data_as(ctypes.c_void_p), 1) == 0
    for n in (1, 8):
        steps = np.full(n, STEPS, dtype=np.uint64)
        out = np.zeros(n * (p.mexp // 32 + 1), dtype=np.uint32)
        for _ in range(2):  # the first also makes the tables
            fake.clear()
            assert L.mtgp64_gpu_pool_jump_polys(pool, 0, steps.ctypes.data_as(ctypes.c_void_p), n,
                                                out.ctypes.data_as(ctypes.c_void_p), None) == 0
        assert len([l for l in fake.log() if l.startswith("launchPowOps")]) == launches, n
    L.mtgp64_gpu_pool_free(pool)


@pytest.mark.gpu
@pytest.mark.parametrize("table", ["mtgp64_fast_110503", "mtgp64_fast_44497"])
def test_polynomials(gpu, orc, table):
    """Few and many at once are the same polynomials, and one of them is the
    skip that it stands for."""
    from mtgp_gb300.api import MTGP64, Pool
    p = load_table(table)[0]
    pool = Pool.create([p], [5])
    steps = np.array([STEPS, 1, 300000, (1 << 40) + (1 << 20) + 3, 1 << 63, 255, 256, 65537,
                      STEPS + 1], dtype=np.uint64)
    many = pool.jump_polys(0, steps).cpu().numpy()
    for n in (1, 3, 8):
        assert np.array_equal(pool.jump_polys(0, steps[:n]).cpu().numpy(), many[:n]), n
    g = MTGP64(p, seed=9)
    g.jump_array(many[2].view(np.uint32))
    o = orc.gen(p, seed=9)
    o.skip(300000)
    assert np.array_equal(g.window()[1:], o.window()[1:])
