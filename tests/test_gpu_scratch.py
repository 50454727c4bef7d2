"""Scratch of the tensor-core FP64 products: what stays allocated after a call."""
import ctypes

import pytest

import native

pytestmark = pytest.mark.gpu


def test_no_room_for_the_planes():
    """The FMA kernel takes over: nothing of the other path may stay allocated beside it."""
    L = native.load()
    taken, keep = ctypes.c_int(1), ctypes.c_int64(-1)
    assert L.shim_oz_no_room(ctypes.byref(taken), ctypes.byref(keep)) == 0, L.shim_last_error()
    assert (taken.value, keep.value) == (0, 0)
