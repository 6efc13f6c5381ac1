"""The library's host code on ``fake_cudart.cpp``: the objects of the build
linked with it in the place of the CUDA runtime, loaded beside the real
library.  Arrays in host memory stand for device memory."""
import ctypes
import glob
import os
import subprocess

import numpy as np

from neuralat_b200 import _lib as L
from neuralat_b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))
HOOK = ctypes.CFUNCTYPE(ctypes.c_int, ctypes.c_char_p, ctypes.c_char_p, ctypes.c_void_p, ctypes.c_long)


class FakeCuda:
    def __init__(self, folder):
        build.build()
        path = os.path.join(str(folder), "libhost.so")
        cuda = os.path.join(os.path.dirname(os.path.dirname(build.nvcc())), "include")
        subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-Wl,-Bsymbolic", "-I", cuda, "-o", path,
                        os.path.join(HERE, "fake_cudart.cpp"), *sorted(glob.glob(os.path.join(build.OBJ_DIR, "*.o"))),
                        "-pthread"], check=True)
        self.lib = ctypes.CDLL(path)
        real = L.lib()
        for name in L.EXPORTED:
            fn = getattr(self.lib, name)
            fn.argtypes, fn.restype = getattr(real, name).argtypes, getattr(real, name).restype
        self.lib.fake_hook.argtypes, self.lib.fake_hook.restype = [HOOK], None
        self.lib.fake_device.argtypes, self.lib.fake_device.restype = [ctypes.c_int], None
        self.on = None       # on(event, kernel or direction, pointer, value) -> CUDA error
        self.launched = []   # kernels of the launches that were accepted
        self.refused = []    # and of those that were not
        self._hook = HOOK(self._tell)
        self.lib.fake_hook(self._hook)

    def _tell(self, event, name, pointer, value):
        event, name = event.decode(), name.decode()
        if event in ("launch", "refused"):
            (self.launched if event == "launch" else self.refused).append(name)
        return int(self.on(event, name, pointer, value) or 0) if self.on else 0

    def device(self, d):
        self.lib.fake_device(d)

    def solve(self, n, m=1, precision=L.PREC_FP32, use_x0=0, restart=200):
        p = L.SolverParams(precision=precision, restart=restart, max_iters=100, max_refine=2, rtol=1e-6, atol=0.0,
                           inner_rtol=1e-3)
        A, b, x = array((n, n)), array((n, m)), array((n, m))
        b[:] = 1
        ws = array(int(self.lib.bem_gmres_workspace_bytes(n, m, ctypes.byref(p))), np.uint8)
        return self.lib.bem_gmres_solve(at(A), n, at(b), m, at(x), use_x0, ctypes.byref(p), at(ws), ws.nbytes, None, None)

    def geometry(self, v, t):
        v, t = np.ascontiguousarray(v, np.float32), np.ascontiguousarray(t, np.int32)
        size = ctypes.c_size_t(0)
        L.check(self.lib.bem_geometry_bytes(at(v), len(v), at(t), len(t), ctypes.byref(size), None))
        g = array(size.value, np.uint8)
        L.check(self.lib.bem_geometry_build(at(v), len(v), at(t), len(t), at(g), g.nbytes, None))
        return g


def array(shape, dtype=np.complex64):
    """Zeros at an address that is a multiple of 256, as the allocators of device memory give them."""
    size = int(np.prod(shape)) * np.dtype(dtype).itemsize
    raw = np.zeros(size + 256, np.uint8)
    first = -raw.ctypes.data % 256
    return raw[first:first + size].view(dtype).reshape(shape)


def at(a):
    return a.ctypes.data
