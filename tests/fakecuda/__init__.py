"""The library's host side on the fake CUDA runtime of fake_cudart.cpp: the
object files of libtlq.so linked with it and loaded in the place of the
library.  For tests of what the host decides; kernels do not run."""
import contextlib
import ctypes as C
import os
import subprocess

from tlaloque_gb300 import build, tlq

HERE = os.path.dirname(os.path.abspath(__file__))


class Fake:
    def __init__(self, path):
        self.lib = C.CDLL(path)
        self.lib.fake_calls.restype = self.lib.fake_bytes.restype = C.c_longlong
        self.lib.fake_launch.restype = C.c_char_p
        self.lib.fake_set_cost.argtypes = [C.c_longlong, C.c_double]

    def reset(self):
        self.lib.fake_reset()

    def calls(self, *names):
        """Calls of these runtime functions since reset (frees of null not counted)."""
        return sum(self.lib.fake_calls(n.encode()) for n in names)

    def bytes(self):
        """Bytes allocated at present (device and page-locked)."""
        return self.lib.fake_bytes()

    def launches(self, name=""):
        """(kernel, grid, device) of the launches since reset whose name holds `name`."""
        out = []
        for i in range(self.lib.fake_launches()):
            g, d = (C.c_uint * 3)(), C.c_int()
            k = self.lib.fake_launch(i, g, C.byref(d)).decode()
            if name in k:
                out.append((k, tuple(g), d.value))
        return out

    def set_cost(self, blocks, ms):
        self.lib.fake_set_cost(blocks, ms)

    def fail(self, name):
        self.lib.fake_fail(name.encode())


def link(folder):
    """Links the fake library into `folder`; its path."""
    objects = [os.path.join(build.BUILD_DIR, os.path.splitext(src)[0] + ".o") for src, _ in build.UNITS]
    build.build(force=not all(map(os.path.exists, objects)))
    out = os.path.join(str(folder), "libtlq_fake.so")
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(build.nvcc()))), "include")
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-Wl,-Bsymbolic", f"-I{cuda}",
                    os.path.join(HERE, "fake_cudart.cpp"), *objects,
                    "-o", out], check=True)
    return out


@contextlib.contextmanager
def loaded(path):
    """The package's bindings on the fake library."""
    before, tlq._lib = tlq._lib, None
    try:
        tlq.load_library(path)
        fake = Fake(path)
        fake.reset()
        yield fake
    finally:
        tlq._lib = before
