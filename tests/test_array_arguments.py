"""Which objects the Python calls take for a ``double *`` argument: numpy
arrays, whatever their layout, and nothing else that merely has a buffer."""
from __future__ import annotations

import array
import ctypes as C

import numpy as np
import pytest


def address(arg):
    return C.cast(arg, C.c_void_p).value


@pytest.mark.parametrize("a", [np.arange(6.0), np.arange(12.0)[::2], np.arange(6.0)[2:], np.arange(6.0).reshape(2, 3).T,
                               np.zeros(0), np.arange(7, dtype=np.int64).view(np.float64)],
                         ids=["plain", "strided", "offset", "transposed", "empty", "viewed"])
@pytest.mark.parametrize("writeable", [True, False])
def test_arrays_of_any_layout(pkg, a, writeable):
    a = a[...]
    a.flags.writeable = writeable
    assert address(pkg._arg(a)) == a.ctypes.data


def test_nothing(pkg):
    assert pkg._arg(None) is None


@pytest.mark.parametrize("a", [bytearray(64), memoryview(bytearray(64)), array.array("d", range(8)), (C.c_double * 8)(),
                               [1.0, 2.0], 3.0], ids=["bytearray", "memoryview", "array", "ctypes", "list", "float"])
def test_other_buffers_are_refused(pkg, a):
    """As they always were: their length is nobody's to check."""
    with pytest.raises(AttributeError):
        pkg._arg(a)
