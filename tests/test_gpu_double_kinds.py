"""The 64-bit [0,1), (0,1] and (0,1) kinds: the two-word core subtracts in
integers, which is exact for tables whose entries are in [1, 2); other tables
take the one-word core.  Shipped tables and one with entries outside [1, 2),
by a plain fill, a split fill and a plan, bit for bit against the reference
loop (mtgp64-fast.h:262-356)."""
import copy

import numpy as np
import pytest
import torch

from mtgp_gb300.params import load_table
from gpu_util import np_bits

pytestmark = pytest.mark.gpu


def params(odd):
    p = copy.copy(load_table("mtgp64dc_fast_11213")[4])
    if odd:
        for k, e in ((1, 0x400), (5, 0x3fe), (9, 0x3ff), (15, 0x001)):
            p.dbl_tmp_tbl[k] = (p.dbl_tmp_tbl[k] & ((1 << 52) - 1)) | (e << 52)
    return p


@pytest.mark.parametrize("kind", [2, 3, 4])
@pytest.mark.parametrize("odd", [False, True])
def test_fills_and_plans(gpu, orc, odd, kind):
    from mtgp_gb300.api import MTGP64, Pool, work_items
    p = params(odd)
    g, o = MTGP64(p, seed=17), orc.gen(p, seed=17)
    for n in (1, 100001, (1 << 20) + 5):
        out = torch.zeros(n, dtype=torch.float64, device="cuda")
        g.fill_into(kind, out)
        assert np.array_equal(np_bits(out.cpu().numpy(), 64), np_bits(o.fill(kind, n), 64)), n
    pool = Pool.create([p], [1, 2, 3], [0] * 3)
    lens = [5000, 1, 200001]
    out = torch.zeros(sum(lens), dtype=torch.float64, device="cuda")
    offs = (np.cumsum(lens) - np.array(lens)) * 8
    pool.plan(work_items([0, 1, 2], [kind] * 3, lens, offs)).launch(out)
    got, at = np_bits(out.cpu().numpy(), 64), 0
    for s, n in enumerate(lens):
        want = np_bits(orc.gen(p, seed=s + 1).fill(kind, n), 64)
        assert np.array_equal(got[at:at + n], want), s
        at += n
