"""Row and column of a pixel as the fusion's closures recover them from its index
(smvs_test_row_and_column) against integer division: narrow and tall images, where
the float product is many rows off, ordinary ones, and the ends of each."""
import numpy as np
import pytest

from sensemap_b200 import _native as N


@pytest.mark.parametrize("width", [1, 2, 3, 7, 31, 64, 640, 1600, 6001, 65537, (1 << 31) - 1])
def test_row_and_column_of_any_pixel(width):
    rng = np.random.default_rng(width)
    last = (1 << 31) - 1
    rows = rng.integers(0, last // width + 1, 2000)
    near = np.concatenate([rows * width + d for d in (-1, 0, 1, width - 1)])
    px = np.concatenate([rng.integers(0, last + 1, 20000), near, [0, width - 1, last]])
    px = px[(px >= 0) & (px <= last)].astype(np.uint32)
    row, col = np.zeros(len(px), np.int32), np.zeros(len(px), np.int32)
    N.check(N.lib().smvs_test_row_and_column(px.ctypes.data, len(px), width, row.ctypes.data, col.ctypes.data))
    np.testing.assert_array_equal(row, px // width)
    np.testing.assert_array_equal(col, px % width)
