"""Destinations of served requests: written by the batch's kernel where they
are aligned memory of the server's device, copied otherwise (host memory,
unaligned addresses, destinations that share memory: the later request wins).
Every byte around them stays as it was.  Exact against the reference loop
(mtgp32-fast.h:149-346, mtgp64-fast.h:148-356)."""
import numpy as np
import pytest
import torch

from mtgp_gb300.params import load_table
from gpu_util import np_bits

pytestmark = pytest.mark.gpu


def test_destinations(gpu, orc):
    from mtgp_gb300.api import Pool, REQUEST_DTYPE, Server
    p32, p64 = load_table("mtgp32_fast_11213")[0], load_table("mtgp64dc_fast_11213")[0]
    n = 24
    a = Pool.create([p32], np.arange(n) + 1, [0] * n)
    b = Pool.create([p64], np.arange(n) + 1, [0] * n)
    srv = Server(a, b, budget_bytes=1 << 26, slots=2, max_batch=64)
    gens = {(0, s): orc.gen(p32, seed=s + 1) for s in range(n)}
    gens.update({(1, s): orc.gen(p64, seed=s + 1) for s in range(n)})
    # (pool, stream, kind, count, place): "device" at that byte offset,
    # "pinned" and "pageable" host memory, "shared" the same device place twice
    spec = []
    for s in range(n):
        for pool in (0, 1):
            w = 4 << pool
            count = int([1, 2, 777, 5000, 150001][(s + pool) % 5])
            spec.append((pool, s, (s + pool) % 5, count, ("device", (s % 3) * w)))
    spec += [(0, 1, 0, 1000, ("device", 2)), (1, 2, 0, 1000, ("device", 4)),
             (0, 3, 2, 4000, ("pinned", 0)), (1, 4, 0, 4000, ("pageable", 0)),
             (0, 5, 0, 3000, ("shared", 0)), (0, 5, 0, 2000, ("shared", 0)),
             (1, 6, 1, 9, ("end", 0))]
    req = np.zeros(len(spec), dtype=REQUEST_DTYPE)
    shared = torch.full((4 * 3000 + 32,), 0xA5, dtype=torch.uint8, device="cuda")
    bufs, want = [], []
    for k, (pool, s, kind, count, (place, off)) in enumerate(spec):
        nb = count * (4 << pool)
        if place == "shared":
            buf, lo = shared, 16
        elif place == "end":  # the last byte of its allocation
            buf = torch.full((max(nb, 2 << 20),), 0xA5, dtype=torch.uint8, device="cuda")
            lo = buf.numel() - nb
        else:
            buf = torch.full((nb + 64,), 0xA5, dtype=torch.uint8,
                             device="cuda" if place == "device" else "cpu")
            buf = buf.pin_memory() if place == "pinned" else buf
            lo = 16 + off
        req[k] = (0,) * len(REQUEST_DTYPE.names)
        for f, v in (("pool", pool), ("stream", s), ("kind", kind), ("count", count),
                     ("dst", buf.data_ptr() + lo)):
            req[f][k] = v
        bufs.append((buf, lo, nb))
        want.append(np_bits(gens[pool, s].fill(kind, count), 32 << pool).view(np.uint8))
    srv.replay(req, np.zeros(len(spec)))
    torch.cuda.synchronize()
    srv.close()
    for k, ((buf, lo, nb), w) in enumerate(zip(bufs, want)):
        got = buf.cpu().numpy()
        place = spec[k][4][0]
        if place == "shared":
            continue
        assert np.array_equal(got[lo:lo + nb], w), spec[k]
        assert (got[:lo] == 0xA5).all() and (got[lo + nb:] == 0xA5).all(), spec[k]
    first, last = [w for k, w in enumerate(want) if spec[k][4][0] == "shared"]
    got = shared.cpu().numpy()
    assert np.array_equal(got[16:16 + last.size], last)
    assert np.array_equal(got[16 + last.size:16 + first.size], first[last.size:])
    assert (got[:16] == 0xA5).all() and (got[16 + first.size:] == 0xA5).all()
