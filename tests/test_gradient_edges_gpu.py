"""The reverse walk where a derivative is infinite or NaN, where an adjoint is zero, and at the ends of a
thread's vector: the specialised kernels (SCI_CUDA_JIT: ready after jit_wait) against the interpreter's
walk, which guards every product, in a context of its own. Equal bits: both evaluate the same partials.
"""
import numpy as np
import pytest

from libsci_b200 import chunk as C

pytestmark = pytest.mark.gpu

SPECIAL = [0.0, -0.0, 1.0, -1.0, np.inf, -np.inf, np.nan, 1e-38, -1e-38, 1e-45, 3e38, 2.0 ** 21, -2.0 ** 21, 0.5]


def expressions(a, b):
    return {
        "root": C.unary("root", a) * b,                                     # 1/0 at a = 0, times a zero b
        "log": C.unary("logarithm", a * a) * b,
        "quotient": a / b,
        "circular": C.unary("sin", a) * C.unary("cos", b) + C.unary("sec", a * b),
        "fused": C.unary("exponential", -a * a) * C.unary("sin", b) + C.unary("logarithm", 1 + a * a),
        "extremes": C.binary("minimum", a, b) * C.unary("tan", a) - C.binary("maximum", a, b),
        "repeated": a * a * a + a,
    }


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("count", [1, 3, 4, 5, 1021, 4096 + 7])
def test_specialised_walk(device, dtype, count, monkeypatch):
    from libsci_b200.device import Device

    rng = np.random.default_rng(count)
    values = []
    for salt in range(2):
        v = rng.standard_normal(count).astype(dtype)
        where = rng.integers(0, count, max(1, count // 3))
        v[where] = np.array(SPECIAL, np.float64)[rng.integers(0, len(SPECIAL), where.size)].astype(dtype)
        values.append(v)
    monkeypatch.setenv("SCI_CUDA_JIT", "0")
    plain = Device(0)
    try:
        got = {}
        for which in (device, plain):
            a, b = (which.array(v) for v in values)
            for name, expression in expressions(a.expression(), b.expression()).items():
                for _ in range(2):  # the first call queues the specialisation
                    value, grads = which.gradient(expression, [a, b])
                    which.jit_wait()
                got.setdefault(name, []).append([g.numpy() for g in grads])
        for name, (special, generic) in got.items():
            for s, g in zip(special, generic):
                assert np.array_equal(np.isnan(s), np.isnan(g)) and np.array_equal(s[~np.isnan(s)], g[~np.isnan(g)]), name
                assert np.array_equal(np.signbit(s[~np.isnan(s)]), np.signbit(g[~np.isnan(g)])), name
    finally:
        plain.close()
