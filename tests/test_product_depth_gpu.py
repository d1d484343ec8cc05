"""Tensor-core products whose depth is cut into pieces (few tiles), and the edges of the tiles, pieces and
K slices, against FP64 with the modes' bounds: |C - C64| <= (u + k 2^-22) |A| |B|, u the rounding of the
mode's operands (2^-7 bf16, 2^-14 two terms, 2^-21 three).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(1, 1, 1), (64, 64, 64), (3, 700, 511), (100, 300, 2000), (128, 128, 512), (129, 127, 513), (255, 129, 4097), (257, 1000, 640),
         (1000, 700, 1300), (300, 260, 6001), (2500, 1200, 300)]


@pytest.mark.parametrize("mode,u", [(0, 2.0 ** -7), (1, 2.0 ** -14), (3, 2.0 ** -21)])
@pytest.mark.parametrize("size", SIZES)
def test_depths(device, mode, u, size):
    m, n, k = size
    rng = np.random.default_rng(k)
    a, b = (rng.uniform(-1, 1, s).astype(np.float32) for s in ((m, k), (k, n)))
    a64, b64 = a.astype(np.float64), b.astype(np.float64)
    da, db = device.array(a.ravel()), device.array(b.ravel())
    first = device.product(da, db, m, n, k, mode).numpy()
    assert (np.abs(first.reshape(m, n) - a64 @ b64) <= (u + k * 2.0 ** -22) * (np.abs(a64) @ np.abs(b64))).all()
    for _ in range(3):  # whichever piece is last, the sum is the same
        assert np.array_equal(device.product(da, db, m, n, k, mode).numpy(), first)


@pytest.mark.parametrize("size", [(100, 300, 2000), (257, 1000, 640), (1000, 700, 1300)])
def test_adjoint_depths(device, size):
    m, n, k = size
    rng = np.random.default_rng(m)
    a, b, g = (rng.uniform(-1, 1, s).astype(np.float32) for s in ((m, k), (k, n), (m, n)))
    da, db = device.product_gradient(*(device.array(v.ravel()) for v in (a, b, g)), m, n, k, 3)
    a, b, g = (v.astype(np.float64) for v in (a, b, g))
    assert (np.abs(da.numpy().reshape(m, k) - g @ b.T) <= (2.0 ** -21 + n * 2.0 ** -22) * (np.abs(g) @ np.abs(b).T)).all()
    assert (np.abs(db.numpy().reshape(k, n) - a.T @ g) <= (2.0 ** -21 + m * 2.0 ** -22) * (np.abs(a).T @ np.abs(g))).all()
