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


def corrections(a, b, target):
    """The corrections that the refinement takes with factors and substitutions by columns in FP32 (numpy)."""
    s, n, _ = a.shape
    lu, rows, every = a.astype(np.float32), np.tile(np.arange(n), (s, 1)), np.arange(s)
    for j in range(n):
        p = j + np.argmax(np.abs(lu[:, j:, j]), axis=1)
        for m in (lu, rows):
            m[every, j], m[every, p] = m[every, p].copy(), m[every, j].copy()
        lu[:, j + 1:, j] /= lu[:, j, j, None]
        lu[:, j + 1:, j + 1:] -= lu[:, j + 1:, j, None] * lu[:, j, None, j + 1:]
    x, r, previous = np.zeros((s, n)), b.copy(), np.full(s, np.inf)
    counts, running = np.zeros(s, int), np.ones(s, bool)
    scale = np.abs(a).sum(axis=2).max(axis=1)
    for _ in range(30):
        d = np.take_along_axis(r, rows, axis=1).astype(np.float32)
        for j in range(n):
            d[:, j + 1:] -= lu[:, j + 1:, j] * d[:, j, None]
        for j in range(n - 1, -1, -1):
            d[:, j] /= lu[:, j, j]
            d[:, :j] -= lu[:, :j, j] * d[:, j, None]
        x[running] += d[running]
        counts[running] += 1
        r = b - np.einsum("sij,sj->si", a, x)
        error = np.abs(r).max(axis=1) / (scale * np.abs(x).max(axis=1) + np.abs(b).max(axis=1))
        running &= (error > target) & (error < 0.5 * previous)
        previous = error
    return counts


def test_corrections(device):
    """The factors of ill-conditioned systems (condition 1e6) are as good as those of the elimination by columns:
    as many corrections on average. A system's count differs by about a half from run to run of the
    rounding, so the means of 120 by 0.065; four times that is the bound."""
    rng, n, s = np.random.default_rng(48), 48, 120
    q1, q2 = (np.linalg.qr(rng.standard_normal((s, n, n)))[0] for _ in range(2))
    a, b = (q1 * np.logspace(0, -6, n)) @ q2, rng.standard_normal((s, n))
    _, _, counts = batch_of(device, a, b)
    assert counts.mean() <= corrections(a, b, 1e-15).mean() + 0.26
    single = [device.solve(device.array(m.ravel()), device.array(v), n, 1, refine=True)[2] for m, v in zip(a, b)]
    assert np.mean(single) <= corrections(a, b, np.sqrt(n) * 2.0 ** -53).mean() + 0.26


@pytest.mark.parametrize("n", [16, 33, 100, 200, 225, 256])
def test_remaining_error(device, n):
    """What is left at the end in diagonally dominant systems. A solution rounded to nearest has a backward error of
    at most 2^-53; the last residual's own rounding is random and adds less than half of that."""
    rng, s = np.random.default_rng(n), 12
    a = rng.standard_normal((s, n, n)) + n * np.eye(n)
    b, g = rng.standard_normal((s, n, 3)), rng.standard_normal((s, n, 3))

    def error(a, b, x):  # in the longest floating point there is
        a, b, x = (v.astype(np.longdouble) for v in (a, b, x))
        r = b - np.einsum("ij,jk->ik", a, x)
        return (np.abs(r).max(axis=0) / (np.abs(a).sum(axis=1).max() * np.abs(x).max(axis=0) + np.abs(b).max(axis=0))).max()

    worst = []
    for m, v, u in zip(a, b, g):
        x, _, y, _, _ = device.solve_gradient(*(device.array(t.ravel()) for t in (m, v, u)), n, 3, refine=True)
        z = device.solve(device.array(m.ravel()), device.array(v[:, 0]), n, 1, refine=True)[0]
        worst += [error(m, v, x.numpy().reshape(n, 3)), error(m.T, u, y.numpy().reshape(n, 3)), error(m, v[:, :1], z.numpy()[:, None])]
    assert max(worst) <= 1.5 * 2.0 ** -53
