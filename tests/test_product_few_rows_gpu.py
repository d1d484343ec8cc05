"""Products and adjoints of few rows and many columns, whose tiles lie along C's columns (two and three terms) or
on single CTAs (one), at the rows, columns and depths where that begins and ends, against FP64: the worst
entry within the mode's operand rounding (2^-7 bf16, 2^-14 two terms, 2^-21 three) plus 2^-22 for each of
the 2048 products that one accumulator takes, and as accurate as the same product of 256 more rows."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(1, 9473, 300), (64, 9473, 64), (65, 9601, 515), (128, 9601, 1024), (128, 9472, 1024), (129, 9601, 1024), (100, 20001, 2100), (17, 9999, 4097)]


@pytest.mark.parametrize("mode,u", [(0, 2.0 ** -7), (1, 2.0 ** -14), (3, 2.0 ** -21)])
@pytest.mark.parametrize("size", SIZES)
def test_few_rows(device, mode, u, size):
    m, n, k = size
    rng = np.random.default_rng(m + k)
    a, b = rng.uniform(-1, 1, (m + 256, k)).astype(np.float32), rng.uniform(-1, 1, (k, n)).astype(np.float32)
    exact = a.astype(np.float64) @ b
    db = device.array(b.ravel())
    few = device.product(device.array(a[:m].ravel()), db, m, n, k, mode).numpy().reshape(m, n)
    many = device.product(device.array(a.ravel()), db, m + 256, n, k, mode).numpy().reshape(m + 256, n)
    scale = np.abs(a[:m]).astype(np.float64) @ np.abs(b)
    assert (np.abs(few - exact[:m]) <= (u + 2048 * 2.0 ** -22) * scale).all()
    rms = [np.sqrt(np.mean((x - exact[:len(x)]) ** 2)) for x in (few, many)]
    assert rms[0] <= 1.25 * rms[1]  # thousands of entries: a few per cent apart at most
