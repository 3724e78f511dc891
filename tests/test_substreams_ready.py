"""A pool of substreams on a stream being captured is refused before anything
is recorded there (its windows would be made by replays of the graph, not by
the call), and a pool of one stream is ready when the call returns."""
import ctypes

import pytest

from mtgp_gb300.params import jump_table, load_table

STREAM = 0x1000


@pytest.fixture(scope="module")
def fake():
    import fake_gpu
    return fake_gpu.load()


def create(fake, bits, count, stream=STREAM):
    p = load_table("mtgp32_fast_11213" if bits == 32 else "mtgp64dc_fast_11213")[0]
    t = jump_table(bits)
    h = ctypes.c_void_p()
    rc = getattr(fake.lib, "mtgp%d_gpu_pool_create_substreams" % bits)(
        ctypes.byref(h), ctypes.byref(p), 5, count, t.ctypes.data_as(ctypes.c_void_p), t.shape[0],
        t.shape[1], stream)
    if h.value:
        getattr(fake.lib, "mtgp%d_gpu_pool_free" % bits)(h)
    return rc


@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("count", [1, 100])
def test_capturing_stream_is_refused(fake, bits, count):
    fake.clear()
    fake.capture(STREAM)
    assert create(fake, bits, count) != 0
    assert not [l for l in fake.log() if "captured" in l]
    fake.clear()
    assert create(fake, bits, count) == 0


@pytest.mark.parametrize("bits", [32, 64])
def test_one_stream_is_ready(fake, bits):
    fake.clear()
    assert create(fake, bits, 1) == 0
    log = fake.log()
    seeded = log.index("launchSeed%d " % bits)
    freed = log.index("cudaDeviceSynchronize")  # pool_free's
    assert "cudaStreamSynchronize" in log[seeded:freed]


@pytest.mark.gpu
def test_relaxed_capture(gpu):
    import torch
    from mtgp_gb300._lib import MTGPError
    from mtgp_gb300.api import Pool
    p, t = load_table("mtgp32_fast_11213")[0], jump_table(32)
    st = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.graph(torch.cuda.CUDAGraph(), stream=st, capture_error_mode="relaxed"):
        with pytest.raises(MTGPError):
            Pool.substreams(p, 5, 3, t, stream=st)
    assert Pool.substreams(p, 5, 3, t, stream=st).windows().shape[0] == 3
