"""``util.pair`` is ``np.broadcast_to(x, (2,))`` in everything but its cost."""
import numpy as np
import pytest

import lentil_gb300 as lg
from lentil_gb300 import util


@pytest.mark.parametrize('x', [3, 2.5, np.float64(0.1), np.int64(7), True, np.float32(0.3), (1, 2), [0.5, 4], (1, 2.5),
                               np.array([1e-3, 2e-3]), np.array([4, 5]), np.array(3.0), np.array([6.0]), [np.float32(1), 2],
                               (np.int64(3), 4.5), np.arange(4.0)[::2]])
def test_pair(x):
    a, b = util.pair(x), np.broadcast_to(x, (2,))
    assert a.dtype == b.dtype and a.shape == b.shape and np.array_equal(a, b)
    assert not a.flags.writeable
    with pytest.raises(ValueError):
        a[0] = 1


def test_pixelscale_is_not_a_way_into_the_callers_array():
    mine = np.array([1e-3, 2e-3])
    w = lg.Pupil(pixelscale=mine)
    with pytest.raises(ValueError):
        w.pixelscale[0] = 5.0
    assert mine.flags.writeable and mine[0] == 1e-3
    mine[1] = 3e-3                            # a view of it, as np.broadcast_to gives
    assert w.pixelscale[1] == 3e-3


def _boundary(x, threshold):
    x = np.asarray(x) > threshold
    rows, cols = np.flatnonzero(x.any(axis=1)), np.flatnonzero(x.any(axis=0))
    return rows[0], rows[-1], cols[0], cols[-1]


@pytest.mark.parametrize('threshold', [0, 0.0, False, 0.5, True, float('nan'), np.array(0), np.array([[0], [1], [0]]),
                                       np.array([0, 0, 0.5, 0])])
@pytest.mark.parametrize('dtype', [bool, float, int])
def test_boundary(dtype, threshold):
    x = np.array([[0, 0, 0, 0], [0, 1, 0, 0], [0, 1, 1, 0]], dtype=dtype)
    try:
        want = _boundary(x, threshold)
    except IndexError:                         # nothing above the threshold
        with pytest.raises(IndexError):
            util.boundary(x, threshold)
        return
    assert util.boundary(x, threshold) == want


@pytest.mark.parametrize('dtype', [bool, float])
def test_boundary_of_a_cube(dtype):
    x = np.zeros((3, 5, 7), dtype=dtype)
    x[1, 2:4, 3:6] = 1
    x[0, 4, 1] = 1
    assert util.boundary(x) == _boundary(x, 0)
