"""Broadcasts and axis folds whose rows are not whole 16-byte vectors: the ends of a row's vectors, rows
that start between boundaries, arrays that start on an odd element, and the lengths at which a fold
changes its step. Against numpy, whose rules these operations follow bit for bit (folds: one rounding
of a double sum, as test_shapes_gpu.py bounds them).
"""
import numpy as np
import pytest

from libsci_b200 import chunk as C

pytestmark = pytest.mark.gpu


def shifted(device, values, shift):
    """A device copy that starts `shift` elements after an aligned address."""
    flat = np.concatenate([np.zeros(shift, values.dtype), values.ravel()])
    return device.array(flat).offset(shift)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("columns", [63, 64, 65, 66, 67, 127, 1023, 1025, 2047, 2048, 2049, 2051, 4099])
@pytest.mark.parametrize("shift", [0, 1])
def test_ragged_rows(device, dtype, columns, shift):
    rng = np.random.default_rng(columns)
    for shape in ((7, columns), (1, columns), (3, 5, columns)):
        x = rng.standard_normal(shape).astype(dtype)
        y = rng.standard_normal(shape).astype(dtype)
        row = rng.standard_normal((1,) * (len(shape) - 1) + (columns,)).astype(dtype)
        column = np.round(rng.standard_normal(shape[:-1] + (1,))).astype(dtype)
        middle = rng.standard_normal(shape[:1] + (1,) * (len(shape) - 2) + (columns,)).astype(dtype)
        d = {k: (shifted(device, v, shift), v.shape) for k, v in
             {"x": x, "y": y, "row": row, "column": column, "middle": middle}.items()}
        for code, names, want in (("where", ("column", "x", "y"), np.where(column != 0, x, y)), ("add", ("column", "row"), column + row),
                                  ("subtract", ("x", "middle"), x - middle), ("multiply", ("x", "y"), x * y),
                                  ("floor", ("x",), np.floor(x))):
            got, shape_got = device.broadcast(code, [d[n] for n in names])
            assert shape_got == want.shape and np.array_equal(got.numpy().reshape(want.shape), want), (code, shape)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("shape", [(1, 64), (3, 511), (3, 512), (3, 513), (9, 1), (64, 3), (65, 4), (7, 8), (8, 7), (129, 33), (2048, 2), (700, 1000),
                                   (6400, 700), (5, 9001)])
def test_axis_lengths(device, dtype, shape):
    rng = np.random.default_rng(shape[0])
    x = rng.standard_normal(shape).astype(dtype)
    for shift in (0, 1):
        array = shifted(device, x, shift)
        for axis in (0, 1):
            wide = x.astype(np.longdouble).sum(axis=axis)
            bound = shape[axis] * 2.0 ** -52 * np.abs(x.astype(np.float64)).sum(axis=axis) + (
                np.spacing(np.abs(wide).astype(np.float32)).astype(np.float64) if dtype == np.float32 else 0.0)
            total = device.reduce_axis(array, shape, axis, C.SUM)[0].numpy()
            assert (np.abs(total.astype(np.longdouble) - wide) <= bound).all()
            assert np.array_equal(device.reduce_axis(array, shape, axis, C.MINIMUM)[0].numpy(), x.min(axis=axis))
            assert np.array_equal(device.reduce_axis(array, shape, axis, C.MAXIMUM)[0].numpy(), x.max(axis=axis))
