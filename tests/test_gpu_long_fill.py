"""Fills around the length from which a generator takes the long shared
buffer, and around that buffer's segments (42 sub-steps of 256 or 128 words):
values, neighbours and the sequence continued by a later fill, against the
reference loop (mtgp32-fast.h:149-346, mtgp64-fast.h:148-356)."""
import numpy as np
import pytest
import torch

from mtgp_gb300.params import load_table
from gpu_util import check_guards, guarded, np_bits

pytestmark = pytest.mark.gpu

CASES = [(32, "mtgp32_fast_11213", 7, 42 * 256), (64, "mtgp64dc_fast_11213", 9, 42 * 128)]


@pytest.mark.parametrize("kind", range(5))
@pytest.mark.parametrize("bits,table,idx,seg", CASES)
def test_lengths(gpu, orc, bits, table, idx, seg, kind):
    from mtgp_gb300.api import MTGP32, MTGP64
    p = load_table(table)[idx]
    g = (MTGP32 if bits == 32 else MTGP64)(p, seed=31)
    o = orc.gen(p, seed=31)
    for n in (16383, 16384, 16385, 2 * seg - 1, 2 * seg, 2 * seg + 1, 3 * seg + 130, 7):
        for off in (0, 1, 3):
            full, view = guarded(n + off, bits, kind)
            g.fill_into(kind, view[off:], n)
            check_guards(full, bits)
            got = np_bits(view[off:off + n].cpu().numpy(), bits)
            assert np.array_equal(got, np_bits(o.fill(kind, n), bits)), (n, off)
