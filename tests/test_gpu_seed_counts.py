"""Pools of any number of streams are seeded like the reference's generators
(mtgp32-fast.c:119-137, mtgp64-fast.c:124-142): around the number of streams
from which a warp stores its streams' words by rows, and around a warp's."""
import numpy as np
import pytest

from mtgp_gb300.params import load_table

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("table", ["mtgp32_fast_11213", "mtgp32_fast_44497",
                                   "mtgp64dc_fast_11213", "mtgp64_fast_110503"])
def test_windows(gpu, orc, table):
    from mtgp_gb300.api import Pool
    bits = int(table[4:6])
    tab = load_table(table)
    for n in (1, 15, 16, 17, 31, 32, 33, 65):
        seeds = (np.arange(n, dtype=np.uint64) * 0x9e3779b1 + 7).astype("u%d" % (bits // 8))
        idx = np.arange(n) % 3
        pool = Pool.create([tab[k] for k in range(3)], seeds, idx)
        assert np.array_equal(pool.windows(), orc.seed_windows(bits, tab, seeds, idx)), n
