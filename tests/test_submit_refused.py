"""What a submit or a plan's launch that failed leaves behind: the windows
jumped ahead of a launch go, by XOR, into slots that have to be zero, so the
next submit must not start from a failed one's slots.  On the host code over a
fake CUDA runtime; the last test on the GPU against the reference loop
(mtgp32-fast.h:149-346)."""
import ctypes

import numpy as np
import pytest

from mtgp_gb300.params import load_table

STREAM = 0x1000


@pytest.fixture(scope="module")
def fake():
    import fake_gpu
    return fake_gpu.load()


@pytest.fixture
def pool(fake):
    fake.clear()
    p = load_table("mtgp32_fast_11213")[0]
    seeds = np.arange(4, dtype=np.uint32)
    idx = np.zeros(4, dtype=np.int32)
    h = ctypes.c_void_p()
    assert fake.lib.mtgp32_gpu_pool_create(ctypes.byref(h), ctypes.byref(p), 1,
                                           idx.ctypes.data_as(ctypes.c_void_p),
                                           seeds.ctypes.data_as(ctypes.c_void_p), 4) == 0
    yield h
    fake.lib.mtgp32_gpu_pool_free(h)


def items():
    """Run starts and chunk offsets: jumps in two launches of parts."""
    from mtgp_gb300._lib import WorkItem
    it = (WorkItem * 2)()
    it[0] = WorkItem(0, 0, 1 << 20, 0, (1 << 18) + 5)
    it[1] = WorkItem(1, 0, 1000, 4 << 20, (1 << 19) + 3)
    return it


def submit(fake, pool, stream=STREAM):
    out = ctypes.create_string_buffer(1)
    return fake.lib.mtgp32_gpu_pool_submit(pool, items(), 2, out, stream)


def cleared_first(log):
    """Whether the jumped windows' slots are zeroed before the first parts."""
    first = next(k for k, l in enumerate(log) if l.startswith("launchJumpParts"))
    return any(l.startswith("cudaMemsetAsync") for l in log[:first])


def test_kept_plan_needs_no_clearing(fake, pool):
    assert submit(fake, pool) == 0
    assert cleared_first(fake.log())
    fake.clear()
    assert submit(fake, pool) == 0
    assert not cleared_first(fake.log())


def test_capturing_stream_is_refused_before_anything_is_recorded(fake, pool):
    assert submit(fake, pool) == 0  # the jump tables are there
    fake.clear()
    fake.capture(STREAM)
    assert submit(fake, pool) != 0
    assert not [l for l in fake.log() if "captured" in l]
    fake.clear()
    assert submit(fake, pool) == 0
    assert [l for l in fake.log() if l.startswith("launchBatch")]


@pytest.mark.parametrize("what,nth", [("launchJumpParts32", 1), ("launchJumpParts32", 2),
                                      ("cudaMemsetAsync", 1), ("launchBatch32", 1),
                                      ("cudaStreamSynchronize", 1)])
def test_failed_submit_leaves_no_jumped_windows(fake, pool, what, nth):
    assert submit(fake, pool) == 0
    fake.clear()
    fake.fail(what, nth)
    assert submit(fake, pool) != 0
    assert any(l == "cudaDeviceSynchronize" for l in fake.log())  # its plan is idle when freed
    fake.clear()
    assert submit(fake, pool) == 0
    assert cleared_first(fake.log())


@pytest.mark.parametrize("what,nth", [("launchJumpParts32", 2), ("cudaMemsetAsync", 1),
                                      ("launchBatch32", 1)])
def test_failed_launch_of_a_kept_plan(fake, pool, what, nth):
    pl = ctypes.c_void_p()
    out = ctypes.create_string_buffer(1)
    assert fake.lib.mtgp32_gpu_pool_plan(pool, items(), 2, ctypes.byref(pl)) == 0
    assert fake.lib.mtgp_gpu_plan_launch(pl, out, STREAM) == 0
    fake.clear()
    fake.fail(what, nth)
    assert fake.lib.mtgp_gpu_plan_launch(pl, out, STREAM) != 0
    fake.clear()
    assert fake.lib.mtgp_gpu_plan_launch(pl, out, STREAM) == 0
    assert cleared_first(fake.log())
    fake.lib.mtgp_gpu_plan_free(pl)


@pytest.mark.gpu
def test_submit_on_a_capturing_stream(gpu, orc):
    import torch
    from mtgp_gb300._lib import MTGPError
    from mtgp_gb300.api import Pool, work_items
    p = load_table("mtgp32_fast_11213")[0]
    pool = Pool.create([p], [1, 2], [0, 0])
    its = work_items([0, 1], [0, 0], [1 << 20, 1000], [0, 4 << 20], [(1 << 18) + 5, (1 << 19) + 3])
    out = torch.zeros((1 << 20) + 1000, dtype=torch.int32, device="cuda")
    gens = [orc.gen(p, seed=1), orc.gen(p, seed=2)]
    st = torch.cuda.Stream()

    def check():
        st.wait_stream(torch.cuda.current_stream())
        pool.submit(its, out, stream=st)
        for g, k in zip(gens, ((1 << 18) + 5, (1 << 19) + 3)):
            g.skip(k)
        want = np.concatenate([gens[0].fill(0, 1 << 20), gens[1].fill(0, 1000)])
        assert np.array_equal(out.cpu().numpy().view(np.uint32), want)

    check()
    torch.cuda.synchronize()
    with torch.cuda.graph(torch.cuda.CUDAGraph(), stream=st, capture_error_mode="relaxed"):
        with pytest.raises(MTGPError):
            pool.submit(its, out, stream=st)
    check()
