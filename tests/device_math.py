"""Host build of the kernels' arithmetic (tests/native/device_math.cpp) for CPU tests."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "lcdrsimulator_b200", "csrc")


def build(out_dir):
    from lcdrsimulator_b200.build import _host_cxx, _nvcc
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(_nvcc()))), "include")
    so = os.path.join(str(out_dir), "device_math.so")
    subprocess.run([_host_cxx(), "-O2", "-std=c++17", "-mfma", "-ffp-contract=off", "-shared", "-fPIC", "-I", CSRC,
                    "-I", cuda, os.path.join(HERE, "native", "device_math.cpp"), "-o", so], check=True)
    return C.CDLL(so)


def ptr(a):
    return a.ctypes.data_as(C.c_void_p)


def nematic(lib, q, iso_cut=1e-9):
    q = np.ascontiguousarray(q, dtype=np.float64)
    out = np.empty((len(q), 4))
    lib.dm_nematic(ptr(q), C.c_longlong(len(q)), C.c_double(iso_cut), ptr(out))
    return out


def chem(lib, q, dx, e, packed):
    """Chemical potential of an FP32 field (5, n, n, n) on cells 2 .. n - 3, e = (L1, L2, L3, cQ, cQ2, cQ3)."""
    n = q.shape[1]
    mu = np.full(q.shape, np.nan, dtype=np.float32)
    lib.dm_chem(ptr(q), n, C.c_double(dx), ptr(np.asarray(e, dtype=np.float64)), int(packed), ptr(mu))
    return mu
