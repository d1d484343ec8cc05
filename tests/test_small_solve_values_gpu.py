"""Small solves at the values and conditions where a shortcut in the factorisation or the residual shows:
infinite entries, ill-conditioned systems (corrections until the stopping rule holds) and the backward
error that is left at the end.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def batch_of(device, matrices, rights):
    """x, backward errors and corrections of one batched launch."""
    orders = [m.shape[0] for m in matrices]
    da, db = [device.array(m.ravel()) for m in matrices], [device.array(v) for v in rights]
    dx = [device.empty(n, np.float64) for n in orders]
    errors, iterations = device.empty(len(orders), np.float64), device.empty(len(orders), np.int32)
    batch = device.solve_batch(orders, *[[v.pointer for v in t] for t in (da, db, dx)], errors, iterations)
    batch.launch()
    made = [v.numpy() for v in dx], errors.numpy(), iterations.numpy()
    batch.close()
    return made


@pytest.mark.parametrize("n", [2, 5, 33, 65, 100, 129, 200, 225, 256])
def test_infinite_pivot(device, n):
    """An infinite entry is its column's pivot, by which the other rows divide to zero: the column's unknown is
    0, the entry's row drops out and the others solve the rest (no NaN)."""
    rng = np.random.default_rng(n)
    row, column = n // 2, n // 3
    a = rng.standard_normal((n, n)) + n * np.eye(n)
    a[[row, column]] = a[[column, row]]  # the rest stays diagonally dominant
    a[row, column] = np.inf
    b = rng.standard_normal(n)
    rest = np.linalg.solve(np.delete(np.delete(a, row, 0), column, 1), np.delete(b, row))
    want = np.insert(rest, column, 0.0)
    x, _, _ = device.solve(device.array(a.ravel()), device.array(b), n, 1, refine=True)
    (y,), _, _ = batch_of(device, [a], [b])
    for got in (x.numpy(), y):  # one correction in FP32 (the error is not a number): its rounding, 2^-24 n
        assert np.abs(got - want).max() <= n * 2.0 ** -24 * np.abs(want).max()
