"""The jump kernel that sorts a polynomial's rows of eight taps by pattern, at
the edges of its layout: no rows, one row, rows of one pattern only, every
pattern, polynomials longer than one chunk of taps, and jumps shared out over
any number of CTAs.  Exact against the reference's tap-by-tap walk
(mtgp32-fast-jump.c:51-79)."""
import numpy as np
import pytest
import torch

from mtgp_gb300.params import load_table

pytestmark = pytest.mark.gpu

TABLES = [(32, "mtgp32_fast_11213", 3), (64, "mtgp64dc_fast_11213", 1),
          (32, "mtgp32_fast_23209", 0), (64, "mtgp64_fast_23209", 5)]


def polys(mexp):
    n = mexp // 32 + 1
    rng = np.random.default_rng(mexp)
    yield "zero", np.zeros(n, np.uint32)
    yield "one word", np.array([0x80000001], np.uint32)
    last = np.zeros(n, np.uint32)
    last[-1] = 1 << (mexp % 32 - 1)
    yield "last tap", last
    yield "one pattern", np.full(n, 0x05050505, np.uint32)
    yield "all taps", np.full(n, 0xffffffff, np.uint32)
    every = np.resize(np.arange(256, dtype=np.uint8), 4 * n).view("<u4")
    yield "every pattern", every.astype(np.uint32)
    yield "longest", rng.integers(0, 2 ** 32, 2 * n, dtype=np.uint64).astype(np.uint32)


@pytest.mark.parametrize("bits,table,idx", TABLES)
def test_patterns(gpu, orc, bits, table, idx):
    from mtgp_gb300.api import MTGP32, MTGP64
    p = load_table(table)[idx]
    for name, poly in polys(p.mexp):
        g = (MTGP32 if bits == 32 else MTGP64)(p, seed=99)
        o = orc.gen(p, seed=99)
        g.jump_array(poly)
        o.jump_words(poly)
        assert np.array_equal(g.window(), o.window()), name


@pytest.mark.parametrize("parts", [1, 2, 5, 8, 31, 32, 40])
@pytest.mark.parametrize("bits,table,idx", TABLES)
def test_shares(gpu, orc, bits, table, idx, parts):
    from mtgp_gb300.api import MTGP32, MTGP64
    p = load_table(table)[idx]
    g = (MTGP32 if bits == 32 else MTGP64)(p, seed=7)
    g.set_tuning("jump_parts", parts)
    n = (1 << 20) + 3
    out = torch.zeros(n, dtype=torch.int32 if bits == 32 else torch.int64, device="cuda")
    g.fill_into(0, out)
    want = orc.gen(p, seed=7).fill(0, n)
    assert np.array_equal(out.cpu().numpy().view(want.dtype), want)
