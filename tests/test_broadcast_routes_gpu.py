"""Broadcasts of ragged rows at the lengths where their form changes (flat index, rows, vectors), against numpy,
and the time of many short rows beside that of the same elements in one row: a form that leaves most of a
block idle on short rows took 25 times as long."""
import ctypes
import time

import numpy as np
import pytest

from libsci_b200 import chunk as C
from libsci_b200.native import check, lib

pytestmark = pytest.mark.gpu


def shifted(device, values, shift):
    return device.array(np.concatenate([np.zeros(shift, values.dtype), values.ravel()])).offset(shift)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("columns", [287, 288, 289, 575, 576, 577, 1023, 1025, 2047, 2048, 2049, 4096])
@pytest.mark.parametrize("shift", [0, 1])
def test_forms(device, dtype, columns, shift):
    rng = np.random.default_rng(columns)
    x, y = (rng.uniform(0.1, 3.0, (11, columns)).astype(dtype) for _ in range(2))
    column, row = np.round(rng.standard_normal((11, 1))).astype(dtype), rng.standard_normal((1, columns)).astype(dtype)
    d = {k: (shifted(device, v, shift), v.shape) for k, v in {"x": x, "y": y, "column": column, "row": row}.items()}
    for code, names, want in (("where", ("column", "x", "y"), np.where(column != 0, x, y)), ("add", ("column", "row"), column + row),
                              ("subtract", ("x", "column"), x - column), ("ceil", ("x",), np.ceil(x))):
        got, shape = device.broadcast(code, [d[n] for n in names])
        assert shape == want.shape and np.array_equal(got.numpy().reshape(shape), want), code
    got, shape = device.broadcast("power", [d["x"], d["column"]])
    want = np.power(x.astype(np.float64), column.astype(np.float64))
    assert (np.abs(got.numpy().reshape(shape) - want) <= 2 * np.spacing(np.abs(want).astype(dtype))).all()


@pytest.mark.parametrize("columns", [65, 129, 255])
def test_short_rows_keep_the_blocks_busy(device, columns):
    rows = 26_000_000 // columns
    x, y, column, one = (device.ones(k) for k in (rows * columns, rows * columns, rows, 1))

    out = device.empty(rows * columns)

    def seconds(shape, operands):
        inputs = (ctypes.c_void_p * 3)(*[a.pointer for a, _ in operands])
        extents = (ctypes.c_uint64 * 6)(*[e for _, own in operands for e in own])
        best = 1e9
        for _ in range(6):
            device.synchronize()
            start = time.perf_counter()
            check(lib.sci_cuda_broadcast(device.handle, 0, C.EXTRA["where"], 2, (ctypes.c_uint64 * 2)(*shape), 3, inputs, extents,
                                         out.pointer), device.handle)
            device.synchronize()
            best = min(best, time.perf_counter() - start)
        return best

    full, whole = (rows, columns), (1, rows * columns)
    table = seconds(full, [(column, (rows, 1)), (x, full), (y, full)])
    line = seconds(whole, [(one, (1, 1)), (x, whole), (y, whole)])
    assert table <= 8 * line  # 3 to 4 as measured
