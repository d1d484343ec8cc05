"""Right-hand sides with columns of zeros: each such column's solution is zero and its error counts as zero,
and the refinement of the columns beside it goes on to the bound of any other solve (a normwise
backward error of at most 1e-14, numpy, FP64).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ORDERS = [1, 33, 100, 225, 256, 257, 600]  # a CTA per group of columns up to 256, blocked beyond


def backward_error(a, b, x):
    return np.abs(b - a @ x).max() / (np.abs(a).sum(axis=1).max() * np.abs(x).max() + np.abs(b).max())


def system(n, width, zeros, seed):
    rng = np.random.default_rng(seed)
    a = rng.standard_normal((n, n)) + n * np.eye(n)
    b = rng.standard_normal((n, width))
    b[:, zeros] = 0.0
    return a, b


def verify(a, b, x, error, iterations):
    for j in range(b.shape[1]):
        if b[:, j].any():
            assert backward_error(a, b[:, j], x[:, j]) <= 1e-14, j
        else:
            assert not x[:, j].any(), j
    assert 0.0 <= error <= 1e-14 and 1 <= iterations <= 60


@pytest.mark.parametrize("width,zeros", [(1, [0]), (3, [1]), (8, [0, 5]), (3, [0, 1, 2]), (65, [64])])
def test_solves(device, width, zeros):
    for n in ORDERS:
        a, b = system(n, width, zeros, n)
        x, error, iterations = device.solve(device.array(a.ravel()), device.array(b.ravel()), n, width, refine=True)
        verify(a, b, x.numpy().reshape(n, width), error, iterations)


@pytest.mark.parametrize("width,zeros", [(1, [0]), (3, [1]), (8, [0, 5])])
def test_adjoints(device, width, zeros):
    for n in ORDERS:
        a, b = system(n, width, [], n)
        g = system(n, width, zeros, n + 1)[1]
        x, _, db, error, iterations = device.solve_gradient(*(device.array(v.ravel()) for v in (a, b, g)), n, width, refine=True)
        verify(a, b, x.numpy().reshape(n, width), error, iterations)
        verify(a.T, g, db.numpy().reshape(n, width), error, iterations)


def test_batch(device):
    a, b = zip(*[system(n, 1, [0] if k % 2 else [], n) for k, n in enumerate((5, 33, 100, 225, 256, 8))])
    orders = [m.shape[0] for m in a]
    da, db = [device.array(m.ravel()) for m in a], [device.array(v.ravel()) for v in b]
    dx = [device.empty(n, np.float64) for n in orders]
    errors, iterations = device.empty(len(a), np.float64), device.empty(len(a), np.int32)
    batch = device.solve_batch(orders, *[[v.pointer for v in t] for t in (da, db, dx)], errors, iterations)
    batch.launch()
    for k, n in enumerate(orders):
        verify(a[k], b[k], dx[k].numpy().reshape(n, 1), errors.numpy()[k], iterations.numpy()[k])
    batch.close()
