"""Axis folds at the lengths and counts where their loads in flight, pieces and waves change, against numpy: sums
within the rounding of a double sum (and of the element), extremes and means of integers exact; and the time of
many short rows and of many pieces beside one long row of the same elements."""
import ctypes
import time

import numpy as np
import pytest

from libsci_b200 import chunk as C
from libsci_b200.native import check, lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("shape", [(3, 64), (50, 65), (9, 127), (9, 128), (9, 129), (5, 511), (5, 512), (5, 513), (5, 1499), (5, 1500), (5, 1501),
                                   (5000, 8200), (3, 20000), (600, 9000), (300001, 5), (300001, 4), (40, 4097, 3)])
def test_folds(device, dtype, shape):
    rng = np.random.default_rng(shape[0])
    x = rng.integers(-1000, 1001, shape).astype(dtype)  # every sum is exact in double
    array = device.array(x.ravel())
    for axis in range(len(shape)):
        total = x.astype(np.float64).sum(axis=axis).ravel()
        assert np.array_equal(device.reduce_axis(array, shape, axis, C.SUM)[0].numpy(), total.astype(dtype))
        assert np.array_equal(device.reduce_axis(array, shape, axis, C.MINIMUM)[0].numpy(), x.min(axis=axis).ravel())
        assert np.array_equal(device.reduce_axis(array, shape, axis, C.MAXIMUM)[0].numpy(), x.max(axis=axis).ravel())
        mean = device.reduce_axis(array, shape, axis, C.AXIS_MEAN)[0].numpy()
        assert np.array_equal(mean, (total / shape[axis]).astype(dtype))


@pytest.mark.parametrize("shape,axis,times", [((800_000, 65), 1, 9), ((800_000, 65), 0, 25)])
def test_times(device, shape, axis, times):
    """Beside the sum of the same elements as 5200 rows of 10000."""
    array, out = device.ones(shape[0] * shape[1]), device.empty(max(shape))

    def seconds(shape, axis):
        extents = (ctypes.c_uint64 * 2)(*shape)
        best = 1e9
        for _ in range(6):
            device.synchronize()
            start = time.perf_counter()
            check(lib.sci_cuda_reduce_axis(device.handle, 0, C.MAXIMUM, array.pointer, 2, extents, axis, out.pointer), device.handle)
            device.synchronize()
            best = min(best, time.perf_counter() - start)
        return best

    assert seconds(shape, axis) <= times * seconds((5200, 10000), 1)  # 5 and 8 as measured
