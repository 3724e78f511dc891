"""A bank's fill around the number of generators up to which a fill takes the
long shared buffer (four per SM; 64-bit also from twelve), and around the lengths that are its segments
(mtgp_device4.cuh kLongBuf): both forms continue every generator exactly
(mtgp32-fast.h:149-346, mtgp64-fast.h:148-356)."""
import numpy as np
import pytest
import torch

from mtgp_gb300.params import load_table
from gpu_util import np_bits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", [0, 2])
@pytest.mark.parametrize("bits,table,seg", [(32, "mtgp32_fast_11213", 42 * 256),
                                            (64, "mtgp64dc_fast_11213", 21 * 128)])
def test_both_buffers(gpu, orc, bits, table, seg, kind):
    from mtgp_gb300.api import Pool
    p = load_table(table)[1]
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    dt = {(32, 0): torch.int32, (32, 2): torch.float32, (64, 0): torch.int64,
          (64, 2): torch.float64}[bits, kind]
    rows = {}
    for n in (4 * sms, 4 * sms + 1, 12 * sms):
        pool = Pool.create([p], np.arange(n) + 1, [0] * n)
        for count in (16383, 16384, 7 * seg, 7 * seg + 1, 5):
            out = torch.empty(n * count, dtype=dt, device="cuda")
            pool.fill(kind, out, count)
            rows.setdefault(count, []).append(out.view(n, count))
    for count, (a, b, c) in rows.items():
        assert torch.equal(a, b[:4 * sms]), count
        assert torch.equal(b, c[:4 * sms + 1]), count
    for s in (0, 4 * sms):
        o = orc.gen(p, seed=s + 1)
        for count, (_, b, _) in rows.items():
            want = np_bits(o.fill(kind, count), bits)
            assert np.array_equal(np_bits(b[s].cpu().numpy(), bits), want), (s, count)
