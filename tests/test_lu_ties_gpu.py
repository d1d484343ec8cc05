"""The panel's pivot choice where candidates tie, vanish or are NaN, against the column algorithm of
linear::factor (decompose.hpp:29-57) restated in numpy: the first strictly larger magnitude in the
current row order is the pivot, a NaN only where it stands at the pivot position, a zero pivot leaves
its column. The matrices are totally unimodular (intervals of ones with the signs of some rows and
columns turned), so every value of any elimination order is -1, 0 or 1: nearly every choice is a tie,
no operation rounds, and rows and factors are equal without a tolerance."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def column_factor(a):
    a = a.copy()
    n = a.shape[0]
    rows = np.arange(n)
    for j in range(n):
        magnitude = np.abs(a[j:, j])
        p = j if np.isnan(magnitude[0]) else j + int(np.argmax(np.where(np.isnan(magnitude), -1, magnitude)))
        if p != j:
            a[[j, p]] = a[[p, j]]
            rows[[j, p]] = rows[[p, j]]
        if a[j, j] != 0:
            a[j + 1:, j] /= a[j, j]
            a[j + 1:, j + 1:] -= a[j + 1:, j, None] * a[j, j + 1:]
    return a, rows


@pytest.mark.parametrize("n", [2, 31, 33, 250, 511, 513, 1025, 2049])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("kind", ["ties", "zeros", "nan"])
def test_pivot_choice(device, n, dtype, kind):
    rng = np.random.default_rng(n)
    ends = np.sort(rng.integers(0, n, (n, 2)), axis=1)
    column = np.arange(n)
    a = ((column >= ends[:, :1]) & (column <= ends[:, 1:])).astype(dtype)
    a *= rng.choice([-1, 1], (n, 1)) * rng.choice([-1, 1], (1, n))
    if kind == "zeros":
        a[:, n // 2:] = a[:, :n - n // 2]  # repeated columns: zero pivots
    if kind == "nan":
        a[n // 2, n - 1] = np.nan  # in the last column, so that the other columns stay numbers
    with np.errstate(all="ignore"):
        lu, order = column_factor(a)
    d = device.array(a.ravel())
    rows = device.factor(d, n, plain=True)
    assert np.array_equal(np.asarray(rows, np.int64), order)
    # the NaN's own column is left out: below a zero pivot, the updates by whole panels multiply its
    # zeros by the NaN where the column algorithm skips them
    compared = n - 1 if kind == "nan" else n
    assert np.array_equal(d.numpy().reshape(n, n)[:, :compared], lu[:, :compared])
