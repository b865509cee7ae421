"""What the allocation-free EDT refuses, and why it says so (decided before any GPU work)."""

import ctypes

from torchmorph_gb300 import _lib


def _call(shape):
    lib = _lib.load()
    buf = ctypes.create_string_buffer(64)  # never read: the shape is refused first
    at = ctypes.addressof(buf)
    st = lib.tm_edt_noalloc(at, _lib.TM_U8, 1, len(shape), _lib.i64_array(shape), at, None, None, None)
    return st, lib.tm_last_error().decode()


def test_refused_shapes_are_named():
    st, why = _call([4, 257, 8])
    assert st == 2 and "256 voxels along axis 1, got 257" in why
    st, why = _call([4, 8, 8, 8])
    assert st == 2 and "2-D or 3-D" in why
