"""Host arrays at the C-ABI: the library's order (first axis fastest) whatever
the caller's layout, no copy where it is that order already, pointers that
keep their array alive."""
import ctypes as C
import gc

import numpy as np
import pytest

from diffusecode_gb300 import _abi
from diffusecode_gb300 import fourier as FR


@pytest.mark.parametrize("shape", [(1, 1, 1), (5, 1, 1), (4, 3, 1), (3, 4, 5), (0, 2, 2)])
@pytest.mark.parametrize("layout", ["C", "F", "strided", "float32"])
def test_flat_in_order(shape, layout):
    v = np.arange(np.prod(shape), dtype=np.float64).reshape(shape)
    a = {"C": np.ascontiguousarray(v), "F": np.asfortranarray(v), "float32": v.astype(np.float32),
         "strided": np.repeat(v, 2, axis=0)[::2]}[layout]
    f = FR._flat_in(a)
    assert f.dtype == np.float64 and f.flags.c_contiguous
    np.testing.assert_array_equal(f, v.reshape(-1, order="F"))
    if layout == "F" and v.size:
        assert np.shares_memory(f, a)


def test_complex_results_are_interleaved_doubles():
    z = FR._out((3, 2, 1), np.complex128)
    p = _abi.dptr(z)
    for k in range(12):
        p[k] = float(k)
    np.testing.assert_array_equal(z.reshape(-1, order="F"), np.arange(0, 12, 2) + 1j * np.arange(1, 12, 2))


def test_pointer_keeps_the_array():
    p = _abi.dptr(np.full(1000, 7.0))
    gc.collect()
    junk = [np.full(1000, -1.0) for _ in range(50)]
    assert p[999] == 7.0 and junk[0][0] == -1.0
    assert not _abi.dptr(None) and not _abi.iptr(None)
    with pytest.raises(AssertionError):
        _abi.dptr(np.zeros(4, np.float32))
    with pytest.raises(AssertionError):
        _abi.dptr(np.zeros((4, 4))[::2, ::2])
    assert isinstance(p, C.POINTER(C.c_double))
