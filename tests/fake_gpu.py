"""The library linked with a CUDA runtime that runs nothing (fake_cudart.cpp), so
that its host code can be tested where there is no GPU: `fake_gpu(monkeypatch,
directory)` points the binding at it and returns (binding, handle of the fake)."""
import ctypes
import os
import subprocess

_built = {}


def build(directory):
    from su2higgs_gb300 import build as b
    if "lib" not in _built:
        b.build()
        out = os.path.join(str(directory), "libsu2gpu_fake.so")
        src = os.path.join(os.path.dirname(os.path.abspath(__file__)), "fake_cudart.cpp")
        cuda = os.path.dirname(os.path.dirname(b.nvcc()))
        objs = [os.path.join(b.BUILD, name + ".o") for name, _, _ in b.UNITS]
        subprocess.run(["g++", "-O1", "-shared", "-fPIC", "-std=c++17", "-Wl,-Bsymbolic", "-I",
                        os.path.join(cuda, "include"), "-o", out, src] + objs, check=True)
        _built["lib"] = out
    return _built["lib"]


class Fake:
    def __init__(self, lib):
        self.lib = lib
        lib.fake_op.restype = ctypes.c_char_p
        lib.fake_live_bytes.restype = ctypes.c_int64
        lib.fake_watched.restype = ctypes.c_uint64
        lib.fake_room.restype = ctypes.c_int64
        lib.fake_room.argtypes = [ctypes.c_uint64]

    def reset(self):
        self.lib.fake_reset()

    def fail(self, what, n):
        """The call `what` after n more successful ones fails."""
        self.lib.fake_fail(what.encode(), n)

    def failed(self, what):
        return bool(self.lib.fake_failed(what.encode()))

    def live_bytes(self):
        return self.lib.fake_live_bytes()

    def watch(self, kernel, arg):
        """Keep argument `arg` (8 bytes) of the kernel's next launches."""
        self.lib.fake_watch(kernel.encode(), arg)

    def room(self):
        """Bytes of device memory from the watched pointer on."""
        return self.lib.fake_room(self.lib.fake_watched())

    def ops(self):
        a, b = ctypes.c_int64(), ctypes.c_int64()
        out = []
        for k in range(self.lib.fake_ops()):
            what = self.lib.fake_op(k, ctypes.byref(a), ctypes.byref(b)).decode()
            out.append((what, a.value, b.value))
        return out


def fake_gpu(monkeypatch, directory):
    from su2higgs_gb300 import gpu
    monkeypatch.setattr(gpu, "LIB_PATH", build(directory))
    monkeypatch.setattr(gpu, "_lib", None)
    fake = Fake(gpu.lib())
    fake.reset()
    return gpu, fake
