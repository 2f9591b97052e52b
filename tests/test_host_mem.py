"""Host pages brought in before a mesh is copied back: what the memory holds stays as it is."""

import ctypes as C

import numpy as np
import pytest

from miniisosurface_gb300 import _lib


@pytest.mark.parametrize("offset,nbytes", [(0, 1), (3, 900), (4095, 2), (0, 1 << 20), (17, (3 << 20) + 5)])
def test_populate_keeps_contents(offset, nbytes):
    lib = _lib.load()
    a = (np.arange(offset + nbytes + 64) % 251).astype(np.uint8)
    want = a.copy()
    # one range with bytes, one empty, one absent
    ptrs = (C.c_void_p * 3)(a.ctypes.data + offset, a.ctypes.data, None)
    assert lib.iso_populate_host(3, ptrs, (C.c_int64 * 3)(nbytes, 0, 10)) == _lib.ISO_OK
    assert np.array_equal(a, want)


def test_populate_refuses_bad_arguments():
    lib = _lib.load()
    assert lib.iso_populate_host(0, None, None) == _lib.ISO_OK
    assert lib.iso_populate_host(1, None, None) != _lib.ISO_OK
    assert lib.iso_populate_host(-1, None, None) != _lib.ISO_OK
