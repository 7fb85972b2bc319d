"""Host arrays that kernels read in place (no GPU): an array off its elements'
alignment is copied, one that is not is passed as it is."""
import numpy as np
import pytest

from ehss_b200.engine import _host_array


@pytest.mark.parametrize('offset', [0, 1, 4, 8])
@pytest.mark.parametrize('dtype', [np.float64, np.int64])
def test_alignment(offset, dtype):
    a = np.frombuffer(np.zeros(24 * 8 + 16, dtype=np.uint8), dtype=dtype, count=24, offset=offset).reshape(8, 3)
    got = _host_array(a, dtype)
    assert got.ctypes.data % 8 == 0 and got.flags.c_contiguous and got.dtype == dtype and got.shape == a.shape
    assert np.shares_memory(got, a) == (a.ctypes.data % 8 == 0)


def test_types_and_strides():
    a = np.arange(12, dtype=np.float32).reshape(4, 3)
    got = _host_array(a[::2], np.float64)
    assert got.dtype == np.float64 and got.flags.c_contiguous and np.array_equal(got, a[::2])
