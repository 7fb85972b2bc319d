"""Forms of a source's arrays that explicit-ray calls take (no GPU): longer than
the rays, one entry for all of them, columns, other types; what does not hold
an entry per ray is refused."""
import numpy as np
import pytest

from ehss_b200.engine import _per_ray, _rows


@pytest.mark.parametrize('a,want', [
    (np.arange(12.).reshape(4, 3), np.arange(9.).reshape(3, 3)), (np.arange(3.), np.tile(np.arange(3.), (3, 1))),
    (np.arange(3.).reshape(1, 3), np.tile(np.arange(3.), (3, 1))), (np.arange(9).reshape(3, 3), np.arange(9.).reshape(3, 3)),
    (np.arange(18.).reshape(6, 3)[::2], np.arange(18.).reshape(6, 3)[::2])])
def test_trace_arrays(a, want):
    got = _per_ray(a, np.float64, (3, 3))
    assert got.flags.c_contiguous and got.flags.aligned and got.dtype == np.float64 and np.array_equal(got, want)


@pytest.mark.parametrize('a', [np.zeros((2, 3)), np.zeros((3, 2)), np.zeros((3, 4)), np.zeros((3, 3, 3))])
def test_trace_arrays_refused(a):
    with pytest.raises(ValueError):
        _per_ray(a, np.float64, (3, 3))


@pytest.mark.parametrize('a', [np.arange(4), np.arange(9), np.arange(4).reshape(4, 1), [0, 1, 2, 3], np.arange(8)[::2] // 2])
def test_query_owners(a):
    assert np.array_equal(_rows(a, np.int64, 4, 1).reshape(-1), np.arange(4))


def test_query_rays():
    a = np.arange(15.).reshape(5, 3)
    assert np.array_equal(_rows(a, np.float64, 4, 3), a[:4]) and np.shares_memory(_rows(a, np.float64, 4, 3), a)
    for bad in (a[:3], np.zeros((4, 2)), np.zeros((4, 4)), np.zeros(12)):
        with pytest.raises(ValueError):
            _rows(bad, np.float64, 4, 3)
