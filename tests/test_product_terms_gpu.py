"""Every product of terms that the split modes keep, exactly: operands u + v 2^-9 + w 2^-18 with u, v, w in
-1, 0, 1 are one term each, their products with small integers are multiples of 2^-18, and every sum stays
below 2^6, so FP32 holds all of it and a lost or rounded term shows whatever the depth (a bound that grows
with the depth lets a product of fewer terms pass). Sizes: whole tiles and ragged ones, depths that are cut
into pieces and segments, few rows of many columns.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(1, 1, 64), (64, 64, 512), (100, 300, 2000), (129, 127, 4097), (257, 1000, 640), (300, 260, 6001), (1000, 700, 1300),
         (1, 9601, 1000), (64, 9600, 2050), (100, 12001, 520), (128, 9728, 4100)]


def pieces(rng, shape, terms):
    """u (sparse, so that sums stay small) + v 2^-9 + w 2^-18."""
    x = np.where(rng.random(shape) < 0.01, rng.choice([-1.0, 1.0], shape), 0.0)
    if terms > 1:
        x += rng.integers(-1, 2, shape) * 2.0 ** -9
    if terms > 2:
        x += rng.integers(-1, 2, shape) * 2.0 ** -18
    return x


def operands(size, left_terms, right_terms):
    m, n, k = size
    rng = np.random.default_rng(m + n + k + 7 * left_terms + right_terms)
    whole = lambda shape: rng.choice([-1.0, 1.0], shape)  # noqa: E731
    a = pieces(rng, (m, k), left_terms) if left_terms else whole((m, k))
    b = pieces(rng, (k, n), right_terms) if right_terms else whole((k, n))
    want = a @ b
    assert np.abs(want).max() < 64.0 and (want * 2.0 ** 18 == np.round(want * 2.0 ** 18)).all()
    return a, b, want


@pytest.mark.parametrize("mode,terms", [(0, (1, 0)), (0, (0, 1)), (1, (2, 0)), (1, (0, 2)), (3, (3, 0)), (3, (0, 3)), (3, (2, 2))])
@pytest.mark.parametrize("size", SIZES)
def test_terms(device, mode, terms, size):
    a, b, want = operands(size, *terms)
    da, db = (device.array(v.astype(np.float32).ravel()) for v in (a, b))
    assert np.array_equal(device.product(da, db, *size, mode).numpy().reshape(want.shape), want.astype(np.float32))


@pytest.mark.parametrize("size", [(100, 300, 2000), (257, 1000, 640), (1000, 700, 1300), (128, 1000, 9600), (9600, 1000, 100)])
def test_adjoint_terms(device, size):
    m, n, k = size
    rng = np.random.default_rng(m)
    g = rng.choice([-1.0, 1.0], (m, n))
    a, b = pieces(rng, (m, k), 3), pieces(rng, (k, n), 3)
    left, right = g @ b.T, a.T @ g
    assert max(np.abs(left).max(), np.abs(right).max()) < 64.0
    da, db = device.product_gradient(*(device.array(v.astype(np.float32).ravel()) for v in (a, b, g)), m, n, k, 3)
    assert np.array_equal(da.numpy().reshape(m, k), left.astype(np.float32))
    assert np.array_equal(db.numpy().reshape(k, n), right.astype(np.float32))
