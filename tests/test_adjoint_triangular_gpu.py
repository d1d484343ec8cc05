"""The adjoint of a solve with an ill-conditioned triangular matrix: substitution alone solves it and its transpose
to a backward error of a few 2^-53, whatever the condition (the bound is the refinement's, 1e-14, numpy, FP64),
while factors of the transpose of their own would not. Orders on both sides of the one-launch form's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def backward_error(a, b, x):
    return (np.abs(b - a @ x).max(axis=0) / (np.abs(a).sum(axis=1).max() * np.abs(x).max(axis=0) + np.abs(b).max(axis=0))).max()


@pytest.mark.parametrize("n", [40, 60, 80, 100, 257])
@pytest.mark.parametrize("width", [1, 3])
def test_upper_triangular(device, n, width):
    for seed in range(8):
        rng = np.random.default_rng(1000 * seed + n)
        a = np.triu(rng.standard_normal((n, n))) * (1.0 if n < 257 else 0.2) + 2.0 * np.eye(n)
        b, g = rng.standard_normal((n, width)), rng.standard_normal((n, width))
        x, da, db, error, _ = device.solve_gradient(*(device.array(v.ravel()) for v in (a, b, g)), n, width, refine=True)
        x, db = x.numpy().reshape(n, width), db.numpy().reshape(n, width)
        assert backward_error(a, b, x) <= 1e-14 and backward_error(a.T, g, db) <= 1e-14 and error <= 1e-14, seed
        scale = (np.abs(db) @ np.abs(x).T).max()
        assert np.abs(da.numpy().reshape(n, n) + db @ x.T).max() <= (width + 1) * 2.0 ** -52 * scale
