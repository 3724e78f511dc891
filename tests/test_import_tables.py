"""A generator that has jumped keeps polynomials of its parameter set.  An
import (mtgp32_gpu_import) of a state with other parameters drops them, one
with the same parameters keeps them, and jumps and split fills after either
are those of the imported state.  On the host code over a fake CUDA runtime,
and on the GPU against the reference loop and the reference's tap-by-tap jump
(mtgp32-fast-jump.c:51-79)."""
import ctypes

import numpy as np
import pytest

from mtgp_gb300.params import MTGP32Params, MTGP64Params, load_table

STEPS = 0x123456789abcdef


def fast(bits, params, window):
    """The reference's generator struct with this window (mtgp32-fast.h:60-88)."""
    n = len(window)
    large = 1 << n.bit_length()
    word = ctypes.c_uint32 if bits == 32 else ctypes.c_uint64

    class Status(ctypes.Structure):
        _fields_ = [("idx", ctypes.c_int), ("size", ctypes.c_int), ("large_size", ctypes.c_int),
                    ("large_mask", ctypes.c_int), ("array", word * large)]

    class Fast(ctypes.Structure):
        _fields_ = [("params", MTGP32Params if bits == 32 else MTGP64Params),
                    ("status", ctypes.POINTER(Status))]

    st = Status(idx=n - 1, size=n, large_size=large, large_mask=large - 1)
    for k in range(n):
        st.array[k] = int(window[k])
    return Fast(params=params, status=ctypes.pointer(st))


@pytest.mark.parametrize("same", [True, False])
def test_polynomials_follow_the_parameters(same):
    import fake_gpu
    fake = fake_gpu.load()
    L = fake.lib
    fake.clear()
    tab = load_table("mtgp32_fast_11213")
    old, new = tab[0], tab[0] if same else tab[1]
    assert tab[0].pos != tab[1].pos
    g = ctypes.c_void_p()
    assert L.mtgp32_gpu_init(ctypes.byref(g), ctypes.byref(old), 1) == 0
    out = ctypes.create_string_buffer(16)

    def polys():
        """chi of the products and of the polynomials that jumps read."""
        fake.clear()
        assert L.mtgp32_gpu_jump_steps(g, STEPS, 0, None) == 0
        assert L.mtgp32_gpu_fill(g, 0, out, 1 << 20, None) == 0
        log = fake.log()
        assert all("D 11213" in l for l in log if l.startswith("launchPowOps"))
        return log, {l.split()[-1] for l in log if "chi" in l or "poly" in l}

    _, first = polys()
    assert len(first) == 1
    assert L.mtgp32_gpu_import(g, ctypes.byref(fast(32, new, np.arange(351)))) == 0
    log, after = polys()
    assert len(after) == 1 and (after == first) == same
    assert any(l.startswith("launchBM32") for l in log) == (not same)
    L.mtgp32_gpu_free(g)


@pytest.mark.gpu
@pytest.mark.parametrize("same", [True, False])
@pytest.mark.parametrize("bits,table", [(32, "mtgp32_fast_11213"), (64, "mtgp64dc_fast_11213")])
def test_jumps_and_fills_after_an_import(gpu, orc, bits, table, same):
    import torch
    from mtgp_gb300._lib import check, lib
    from mtgp_gb300.api import MTGP32, MTGP64
    from gpu_util import np_bits
    tab = load_table(table)
    old, new = tab[0], tab[0] if same else tab[1]
    dt = torch.int32 if bits == 32 else torch.int64
    seq = orc.gen(new, seed=1).fill(0, 2 * 11213 + 64)
    deg, chi = orc.minpoly((seq & 1).astype(np.uint8))
    poly = orc.powxmod(STEPS, chi, deg).view(np.uint32)[:11213 // 32 + 1]
    for tune in ((), (("jump_parts", -1),)):
        g = (MTGP32 if bits == 32 else MTGP64)(old, seed=3)
        for k, v in tune:
            g.set_tuning(k, v)
        out = torch.zeros((1 << 22) + 1, dtype=dt, device="cuda")
        g.jump_steps(STEPS)
        g.fill_into(0, out[:(1 << 20) + 5])
        torch.cuda.synchronize()
        o = orc.gen(new, seed=77)
        check(getattr(lib(), "mtgp%d_gpu_import" % bits)(
            g.h, ctypes.byref(fast(bits, new, o.window()))))
        for step in ("old length", "jump", "skip", "new length"):
            if step == "jump":
                g.jump_steps(STEPS)
                o.jump_words(poly)
            elif step == "skip":
                g.skip((1 << 22) + 12345)
                o.skip((1 << 22) + 12345)
            n = (1 << 20) + 5 if step == "old length" else (1 << 22) + 1
            g.fill_into(0, out[:n])
            assert np.array_equal(np_bits(out[:n].cpu().numpy(), bits), o.fill(0, n)), step
