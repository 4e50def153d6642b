"""Sizes that the convolution block's kernels do not index: the C entries refuse them and
the module keeps its layers."""
import ctypes

import pytest

from dtvb200 import _lib, conv

PLANE = [(46341, 46341), (65536, 32768)]  # 2^31 voxels or more, each axis below 2^24


@pytest.mark.parametrize("x,y", PLANE)
def test_entries_refuse_large_planes(x, y):
    L = _lib.load()
    buf = (ctypes.c_char * 64)()  # not read: the size is refused first
    p = ctypes.c_void_p((ctypes.addressof(buf) + 15) // 16 * 16)
    three = (ctypes.c_void_p * 3)(p, p, p)
    none = (ctypes.c_void_p * 3)(p, p, None)
    st = (ctypes.c_int64 * 15)()
    size = _lib.ivec((x, y, 1))
    assert L.dtv_conv_block(p, three, st, three, p, p, p, size, 1, 16, p, None) == 1
    assert L.dtv_conv_block_backward(p, p, three, st, p, p, p, p, p, three, st, none, size, 1, 16, p,
                                     None) == 1


def test_fits():
    assert all(not conv._fits((1, 1, 1, y, x)) for x, y in PLANE)
    assert conv._fits((1, 1, 1, 46340, 46340))
    assert not conv._fits((1, 1, 1, 1, 1 << 24)) and conv._fits((1, 1, 1, 1, (1 << 24) - 1))
    assert not conv._fits((2, 1, 2048, 1024, 1024)) and conv._fits((1, 1, 2048, 1024, 1024))
