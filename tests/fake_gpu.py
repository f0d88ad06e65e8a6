"""The library linked with a CUDA runtime that runs nothing (tests/native/fake_cudart.cpp), for CPU tests of what the
host side allocates, uploads and launches."""
import contextlib
import ctypes as C
import os
import subprocess

import lcdrsimulator_b200 as ldg

HERE = os.path.dirname(os.path.abspath(__file__))


_built = None


def build(out_dir):
    """The library's path; one copy for the process."""
    global _built
    if _built is not None:
        return _built
    from lcdrsimulator_b200.build import LIB, LIB_SOURCES, _host_cxx, _nvcc, build as build_lib
    build_lib()
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(_nvcc()))), "include")
    so = os.path.join(str(out_dir), "libldg_fake.so")
    objs = [os.path.join(LIB, s.replace(".cu", ".o")) for s in LIB_SOURCES]
    subprocess.run([_host_cxx(), "-O1", "-std=c++17", "-shared", "-fPIC", "-I", cuda,
                    os.path.join(HERE, "native", "fake_cudart.cpp"), *objs, "-Wl,-Bsymbolic", "-Wl,--no-undefined",
                    "-lgomp", "-o", so], check=True)
    _built = so
    return so


class Launch:
    def __init__(self, lib, i):
        self.name = lib.fk_name(i).decode()
        self.device = lib.fk_device(i)
        self.grid = lib.fk_grid(i)  # blocks along x
        self.arg = [lib.fk_arg(i, a) for a in range(10)]


class FakeGpu:
    def __init__(self, lib):
        self.lib = lib
        lib.fk_name.restype = C.c_char_p
        lib.fk_arg.restype = C.c_uint64
        lib.fk_is_live.argtypes = [C.c_void_p]

    def fail_malloc(self, n):
        """The n-th allocation from now fails (0: none)."""
        self.lib.fk_fail_malloc(n)

    def pending(self):
        """Operations of the default stream that nothing has waited for."""
        return self.lib.fk_pending()

    def live(self):
        return self.lib.fk_live()

    def is_live(self, p):
        return bool(self.lib.fk_is_live(p))

    def elapsed(self, ms):
        self.lib.fk_elapsed((C.c_float * len(ms))(*ms), len(ms))

    def set_device(self, d):
        self.lib.fk_set_device(d)

    def launches(self, part, start=0):
        return [x for x in (Launch(self.lib, i) for i in range(start, self.lib.fk_launches())) if part in x.name]

    def count(self):
        return self.lib.fk_launches()


@contextlib.contextmanager
def use(so):
    """The package bound to the fake library."""
    path, lib = ldg._LIB_PATH, ldg._lib
    ldg._LIB_PATH, ldg._lib = so, None
    try:
        g = FakeGpu(ldg.load_library())
        g.lib.fk_reset()
        yield g
    finally:
        ldg._LIB_PATH, ldg._lib = path, lib
