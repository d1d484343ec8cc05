"""Systems of order 256 or less, solved by one CTA each: the edges of its 32-column blocks, of the sizes
that change its launch or keep columns in registers, and pivoting that moves rows, ties or skips.

The bound is the refinement's own: a normwise backward error of at most 1e-14 (numpy, FP64).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ORDERS = [1, 2, 3, 31, 32, 33, 63, 64, 65, 95, 96, 97, 127, 128, 129, 151, 152, 153, 191, 192, 193, 223, 224, 225, 241, 255, 256]


def matrix(kind, n, rng):
    g = rng.standard_normal((n, n))
    if kind == "dominant":
        return g + n * np.eye(n)
    if kind == "gaussian":
        return g
    if kind == "reversed":  # every pivot at the far end
        return (g * 1e-3 + n * np.eye(n))[::-1].copy()
    if kind == "ties":  # columns of equal magnitudes
        return np.where(g > 0, 1.0, -1.0) + 2 * n * np.eye(n)[rng.permutation(n)]
    return (g + n * np.eye(n)) * 1e-31


def backward_error(a, b, x):
    return np.abs(b - a @ x).max() / (np.abs(a).sum(axis=1).max() * np.abs(x).max() + np.abs(b).max())


@pytest.mark.parametrize("kind", ["dominant", "gaussian", "reversed", "ties", "tiny"])
def test_batched_orders(device, kind):
    rng = np.random.default_rng(len(kind))
    a = [matrix(kind, n, rng) for n in ORDERS]
    b = [rng.standard_normal(n) for n in ORDERS]
    da, db = [device.array(m.ravel()) for m in a], [device.array(v) for v in b]
    dx = [device.empty(n, np.float64) for n in ORDERS]
    errors, iterations = device.empty(len(ORDERS), np.float64), device.empty(len(ORDERS), np.int32)
    batch = device.solve_batch(ORDERS, [v.pointer for v in da], [v.pointer for v in db], [v.pointer for v in dx], errors,
                               iterations)
    batch.launch()
    for k, n in enumerate(ORDERS):
        assert backward_error(a[k], b[k], dx[k].numpy()) <= 1e-14, n
    assert (errors.numpy() <= 1e-14).all() and (iterations.numpy() <= 30).all()
    batch.close()


@pytest.mark.parametrize("width", [1, 2, 3, 4, 5, 16, 65])
@pytest.mark.parametrize("kind", ["dominant", "gaussian"])
def test_calls(device, width, kind):
    rng = np.random.default_rng(width)
    for n in (1, 5, 32, 33, 64, 97, 128, 200, 224, 225, 256, 257):
        a, b = matrix(kind, n, rng), rng.standard_normal((n, width))
        x, error, iterations = device.solve(device.array(a.ravel()), device.array(b.ravel()), n, width, refine=True)
        x = x.numpy().reshape(n, width)
        worst = max(backward_error(a, b[:, j], x[:, j]) for j in range(width))
        assert worst <= 1e-14 and error <= 1e-14 and 1 <= iterations <= 30, (n, worst, error)


@pytest.mark.parametrize("width", [1, 3, 8])
def test_adjoint_calls(device, width):
    rng = np.random.default_rng(width)
    for n in (1, 31, 64, 96, 129, 200, 224, 241, 256):
        a, b, g = matrix("dominant", n, rng), rng.standard_normal((n, width)), rng.standard_normal((n, width))
        x, da, db, error, _ = device.solve_gradient(*(device.array(v.ravel()) for v in (a, b, g)), n, width, refine=True)
        x, db = x.numpy().reshape(n, width), db.numpy().reshape(n, width)
        worst = max(max(backward_error(a, b[:, j], x[:, j]), backward_error(a.T, g[:, j], db[:, j])) for j in range(width))
        assert worst <= 1e-14 and error <= 1e-14, (n, worst, error)
        want = -db @ x.T  # the outer product of what came back: its rounding only
        assert np.abs(da.numpy().reshape(n, n) - want).max() <= (width + 1) * 2.0 ** -52 * (np.abs(db) @ np.abs(x).T).max(), n


def test_adjoint_over_its_inputs(device):
    """lambda written over the right-hand side: X is still the right-hand side's solution."""
    import ctypes

    from libsci_b200.native import SolveReport, check, lib

    rng, n = np.random.default_rng(7), 100
    a, b, g = matrix("dominant", n, rng), rng.standard_normal(n), rng.standard_normal(n)
    da, db, dg, dx = device.array(a.ravel()), device.array(b), device.array(g), device.empty(n, np.float64)
    check(lib.sci_cuda_solve_gradient(device.handle, 1, 1, da.pointer, db.pointer, dg.pointer, dx.pointer, None, db.pointer, n, 1,
                                      ctypes.byref(SolveReport())), device.handle)
    assert backward_error(a, b, dx.numpy()) <= 1e-14 and backward_error(a.T, g, db.numpy()) <= 1e-14
