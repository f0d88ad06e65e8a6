"""Argument checks of the convolutions' scratch sizes (no GPU)."""
import ctypes as C


def test_scratch_size_of_no_shape(lib):
    from lcdrsimulator_b200.surrogate.conv import SgShape
    f = lib.sg_conv3d_bwd_ws
    f.argtypes, f.restype = [C.POINTER(SgShape)], C.c_longlong
    assert f(None) == 0
    assert f(C.byref(SgShape(1, 8, 0, 8, 32, 32))) == 0
    assert f(C.byref(SgShape(1, 8, 8, 8, 32, -16))) == 0
    assert f(C.byref(SgShape(1, 8, 8, 8, 32, 32))) >= 512 * 32 * 2 + 32 * 27 * 32 * 2
