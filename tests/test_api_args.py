"""The Python side of a call: which objects stand for an address, and the packed argument structs."""
import numpy as np
import pytest

from relux_b200 import api, lib as L


def test_arrays_and_plain_integers_are_addresses():
    a = np.zeros(8, np.float32)
    assert api._ptr(a) == a.ctypes.data and api._ptr(a[2:]) == a.ctypes.data + 8
    assert api._ptr(0x7f0000001000) == 0x7f0000001000 and api._ptr(None) is None


@pytest.mark.parametrize("scalar", [np.int64, np.uint64, np.intp, np.int32])
def test_numpy_integer_scalars_are_refused(scalar):
    """An element of an int64 array of device addresses is neither an array nor an int: it has an __array_interface__ whose
    data is the scalar object itself."""
    p = scalar(0x10000000)
    with pytest.raises(AttributeError):
        api._ptr(p)
    pool = api.Pool.__new__(api.Pool)
    pool.kind = L.POOL_GQA
    with pytest.raises(AttributeError):
        pool._pack_append(0, p, 0x10000000, 1, None, None, L.LAYOUT_TOKEN_MAJOR, True, L.DTYPE_BF16)
    with pytest.raises(AttributeError):
        pool._pack_attn(0, 1, 0x10000000, None, 0x10000000, 8, 128, 1.0, 1, 0, True, L.ATTN_FAST, p, None, None, L.LAYOUT_TOKEN_MAJOR,
                        L.LAYOUT_TOKEN_MAJOR, L.DTYPE_BF16, L.DTYPE_F32)
