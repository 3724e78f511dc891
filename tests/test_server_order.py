"""A server starts on pools whose windows may still be on their way on the
stream that they were made on; its own streams wait for no other.  On the host
code over a fake CUDA runtime: the device is waited for before a batch can
run.  On the GPU: a server made while its pool's jumps are queued behind other
work."""
import ctypes

import numpy as np
import pytest

from mtgp_gb300.params import jump_table, load_table


def test_create_waits_for_the_pools():
    import fake_gpu
    fake = fake_gpu.load()
    L = fake.lib
    fake.clear()
    p = load_table("mtgp32_fast_11213")[0]
    seeds = np.zeros(1, dtype=np.uint32)
    idx = np.zeros(1, dtype=np.int32)
    pool, srv = ctypes.c_void_p(), ctypes.c_void_p()
    assert L.mtgp32_gpu_pool_create(ctypes.byref(pool), ctypes.byref(p), 1,
                                    idx.ctypes.data_as(ctypes.c_void_p),
                                    seeds.ctypes.data_as(ctypes.c_void_p), 1) == 0
    fake.clear()
    assert L.mtgp_server_create(ctypes.byref(srv), pool, None, 1 << 20, 1, 16) == 0
    assert "cudaDeviceSynchronize" in fake.log()
    L.mtgp_server_destroy(srv)
    L.mtgp32_gpu_pool_free(pool)


@pytest.mark.gpu
def test_pool_still_in_the_making(gpu, orc):
    import torch
    from mtgp_gb300.api import Pool, REQUEST_DTYPE, Server
    p, table = load_table("mtgp32_fast_11213")[0], jump_table(32)
    n, count = 64, 5000
    ready = Pool.substreams(p, 1234, n, table)
    ready.fill(0, torch.empty(n * count, dtype=torch.int32, device="cuda"), count)
    want = torch.empty(n * count, dtype=torch.int32, device="cuda")
    ready.fill(0, want, count)  # the second `count` values of each stream
    torch.cuda.synchronize()
    st = torch.cuda.Stream()
    busy = torch.zeros(1 << 28, dtype=torch.uint8, device="cuda")
    with torch.cuda.stream(st):
        out = torch.full((n * count,), -1, dtype=torch.int32, device="cuda")
        st.synchronize()
        for _ in range(50):
            busy.add_(1)
        pool = Pool.substreams(p, 1234, n, table)
        srv = Server(pool, None, budget_bytes=1 << 26, slots=2, max_batch=64)
        req = np.zeros(n, dtype=REQUEST_DTYPE)
        req["stream"] = np.arange(n)
        req["skip"] = count
        req["count"] = count
        req["dst"] = out.data_ptr() + 4 * count * np.arange(n)
        srv.replay(req, np.zeros(n))
        torch.cuda.synchronize()
    assert torch.equal(out, want)
    o = orc.gen(p, seed=1234)
    o.skip(count)
    assert np.array_equal(out[:count].cpu().numpy().view(np.uint32), o.fill(0, count))
    srv.close()
