"""The library's host code over a fake CUDA runtime (fake_cuda.cpp): builds it
once per run and gives the C ABI with a log of what was queued."""
import ctypes
import os
import subprocess
import tempfile

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "mtgp_gb300", "csrc")
SOURCES = ["host.cpp", "plan.cpp", "single.cpp", "pool_api.cpp", "server.cpp", "plan_core.cpp",
           "gf2.cpp"]
_lib = []


class FakeGPU:
    def __init__(self, lib):
        from mtgp_gb300._lib import SIGS
        self.lib = lib
        for name, (res, args) in SIGS.items():
            f = getattr(lib, name, None)
            if f is not None:
                f.restype, f.argtypes = res, args
        lib.fake_fail.argtypes = [ctypes.c_char_p, ctypes.c_int]
        lib.fake_capture.argtypes = [ctypes.c_void_p]

    def clear(self):
        self.lib.fake_clear()

    def log(self):
        n = self.lib.fake_log(None, 0)
        buf = ctypes.create_string_buffer(n + 1)
        self.lib.fake_log(buf, n + 1)
        return buf.value.decode().splitlines()

    def fail(self, name, nth=1):
        self.lib.fake_fail(name.encode(), nth)

    def capture(self, stream):
        self.lib.fake_capture(stream)


def load():
    if not _lib:
        cuda = os.path.dirname(os.path.dirname(os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")))
        d = tempfile.mkdtemp(prefix="fake_gpu")
        so = os.path.join(d, "libfake.so")
        objs, procs = [], []
        for s in [os.path.join(CSRC, f) for f in SOURCES] + [os.path.join(HERE, "fake_cuda.cpp")]:
            objs.append(os.path.join(d, os.path.basename(s) + ".o"))
            procs.append(subprocess.Popen(["g++", "-O1", "-std=c++17", "-fPIC", "-I",
                                           os.path.join(cuda, "include"), "-c", s, "-o", objs[-1]]))
        assert all(p.wait() == 0 for p in procs)
        subprocess.check_call(["g++", "-shared", "-pthread", "-Wl,-Bsymbolic", "-o", so] + objs)
        _lib.append(FakeGPU(ctypes.CDLL(so)))
    return _lib[0]
