"""Submits of one pool refill the plan of the one before (and several threads
at once make their own): growing and shrinking batches, a refused batch in
between, and four threads on streams of their own give the reference loop's
values (mtgp32-fast.h:149-346, mtgp64-fast.h:148-356)."""
import threading

import numpy as np
import pytest
import torch

from mtgp_gb300.params import load_table
from gpu_util import np_bits

pytestmark = pytest.mark.gpu

CASES = [(32, "mtgp32_fast_11213"), (64, "mtgp64dc_fast_11213")]
DT = {32: torch.int32, 64: torch.int64}


def items(streams, counts, bits, skips=None):
    from mtgp_gb300.api import work_items
    c = np.asarray(counts, dtype=np.int64)
    return work_items(streams, np.zeros(len(c), int), c, (np.cumsum(c) - c) * (bits // 8), skips)


@pytest.mark.parametrize("bits,table", CASES)
def test_batches_of_any_size_in_turn(gpu, orc, bits, table):
    from mtgp_gb300._lib import MTGPError
    from mtgp_gb300.api import Pool
    p = load_table(table)[2]
    pool = Pool.create([p], np.arange(40) + 1, [0] * 40)
    gens = [orc.gen(p, seed=s + 1) for s in range(40)]
    rng = np.random.default_rng(bits)
    for rnd, n in enumerate((1, 40, 3, 40, 2)):
        streams = rng.permutation(40)[:n]
        counts = rng.integers(1, 5000, n)
        skips = np.where(rng.random(n) < 0.3, rng.integers(1, 1 << 18, n), 0)
        if rnd == 3:
            counts[0] = 700001  # cut into jumped chunks
        out = torch.zeros(int(counts.sum()), dtype=DT[bits], device="cuda")
        pool.submit(items(streams, counts, bits, skips), out)
        got, at = np_bits(out.cpu().numpy(), bits), 0
        for s, c, k in zip(streams, counts, skips):
            gens[s].skip(int(k))
            assert np.array_equal(got[at:at + c], gens[s].fill(0, int(c))), (rnd, s)
            at += c
        with pytest.raises(MTGPError):
            pool.submit(items([99], [10], bits), out)


@pytest.mark.parametrize("bits,table", CASES)
def test_threads(gpu, orc, bits, table):
    from mtgp_gb300.api import Pool
    p = load_table(table)[0]
    pool = Pool.create([p], np.arange(8) + 1, [0] * 8)
    outs, fails = {}, []

    def work(t):
        try:
            st = torch.cuda.Stream()
            for r in range(6):
                counts = [1000 + 100 * t + r, 333]
                out = torch.zeros(sum(counts), dtype=DT[bits], device="cuda")
                st.wait_stream(torch.cuda.current_stream())
                pool.submit(items([2 * t, 2 * t + 1], counts, bits), out, stream=st)
                outs[t, r] = (counts, out)
        except Exception as e:  # noqa: BLE001
            fails.append(e)

    ts = [threading.Thread(target=work, args=(t,)) for t in range(4)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not fails
    for t in range(4):
        g = [orc.gen(p, seed=2 * t + 1), orc.gen(p, seed=2 * t + 2)]
        for r in range(6):
            counts, out = outs[t, r]
            got = np_bits(out.cpu().numpy(), bits)
            assert np.array_equal(got[:counts[0]], g[0].fill(0, counts[0])), (t, r)
            assert np.array_equal(got[counts[0]:], g[1].fill(0, counts[1])), (t, r)
