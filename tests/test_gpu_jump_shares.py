"""Jumps ahead of a plan's launch, shared by any number of CTAs (tuning knob
jump_parts): even, uneven and single units of the sorted kernel's patterns, and
of the longer exponents' chunks of taps, some parts without any; jumps alone
and chunk offsets behind a run start.  Exact against the reference loop
(mtgp32-fast.h:149-346, mtgp64-fast.h:148-356)."""
import numpy as np
import pytest
import torch

from mtgp_gb300.params import load_table
from gpu_util import np_bits

pytestmark = pytest.mark.gpu

SKIP = {11213: 1 << 17, 23209: 1 << 17, 44497: 1 << 21}


@pytest.mark.parametrize("parts", [1, 2, 5, 8, 31, 32, 40])
@pytest.mark.parametrize("table", ["mtgp32_fast_11213", "mtgp64dc_fast_11213",
                                   "mtgp32_fast_23209", "mtgp64_fast_23209",
                                   "mtgp32_fast_44497", "mtgp64_fast_44497"])
def test_parts(gpu, orc, table, parts):
    from mtgp_gb300.api import Pool, work_items
    bits, p = int(table[4:6]), load_table(table)[1]
    skip = SKIP[p.mexp]
    pool = Pool.create([p], [3, 4], [0, 0])
    pool.set_tuning("jump_parts", parts)
    # stream 0: a run start, then chunks cut from it; stream 1: a jump alone
    long = 2 * skip + 77 if p.mexp < 44497 else 5000
    pool.set_tuning("split_chunk", skip)
    counts, skips = [long, 1000], [skip + 5, 3 * skip + 12345]
    out = torch.zeros(sum(counts), dtype=torch.int32 if bits == 32 else torch.int64, device="cuda")
    items = work_items([0, 1], [0, 0], counts, [0, long * (bits // 8)], skips)
    gens = [orc.gen(p, seed=3), orc.gen(p, seed=4)]
    for _ in range(2):  # the slots are zeroed by the launch before
        pool.submit(items, out)
        got, at = np_bits(out.cpu().numpy(), bits), 0
        for g, c, k in zip(gens, counts, skips):
            g.skip(k)
            assert np.array_equal(got[at:at + c], g.fill(0, c))
            at += c
