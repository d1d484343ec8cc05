"""Gradients of programs whose length and functions change the specialised kernel's registers and walk (11 to 28
nodes), against the interpreter's walk in a context of its own: equal bits, special values included. And the
time of a 14-node program of sines and cosines beside one of 8 nodes: with the registers of four blocks per SM
it took 4.9 times as long, most of it spilled values."""
import ctypes
import time

import numpy as np
import pytest

from libsci_b200 import chunk as C
from libsci_b200.native import check, lib

pytestmark = pytest.mark.gpu


def expressions(a, b, c):
    u = C.unary
    mixed = u("exponential", -a * a) * u("sin", b) + u("logarithm", 1 + c * c)
    trig = u("sin", a * b) * u("cos", b * c) * u("sin", c) + u("cos", a) * u("sin", b) - u("tan", a * 0.1) * c
    long = mixed + u("cos", a * b) * u("root", 2 + c * c) - u("tanh", a + b) * c + u("sin", c * a) * u("exponential", -b * b)
    return {
        "short": mixed,
        "mixed": mixed + u("tanh", a * b) * c,
        "polynomial": (a - b) * (b - c) * (c - a) + a * a * b / (c * c + 1) - a * b,
        "root": mixed + u("cos", a * b) * u("root", 2 + c * c),
        "trig": trig,
        "arithmetic": ((a * b + c) * (a - b) - (b * c + a) * (b - c)) * (a * c + b) / (a * a + b * b + c * c + 1) - a * b * c,
        "long": long,
        "longer": long + (a - b) * (b - c) * u("cos", c),
    }


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("count", [5, 4103])
def test_programs(device, dtype, count, monkeypatch):
    from libsci_b200.device import Device

    rng = np.random.default_rng(count)
    values = []
    for _ in range(3):
        v = rng.standard_normal(count).astype(dtype)
        where = rng.integers(0, count, max(1, count // 5))
        v[where] = rng.choice([0.0, -0.0, 1.0, np.inf, -np.inf, np.nan, 1e-38, 3e38, -2.0 ** 21], where.size).astype(dtype)
        values.append(v)
    monkeypatch.setenv("SCI_CUDA_JIT", "0")
    plain = Device(0)
    try:
        got = {}
        for which in (device, plain):
            arrays = [which.array(v) for v in values]
            for name, expression in expressions(*(x.expression() for x in arrays)).items():
                for stored in (False, True):
                    for _ in range(2):  # the first call queues the specialisation
                        _, grads = which.gradient(expression, arrays, stored=stored)
                        which.jit_wait()
                    got.setdefault((name, stored), []).append([g.numpy() for g in grads])
        for name, (special, generic) in got.items():
            for s, g in zip(special, generic):
                assert np.array_equal(np.isnan(s), np.isnan(g)) and np.array_equal(s[~np.isnan(s)], g[~np.isnan(g)]), name
    finally:
        plain.close()


def test_long_programs_keep_their_values(device):
    n = 1 << 23
    rng = np.random.default_rng(0)
    arrays = [device.array(rng.standard_normal(n).astype(np.float32)) for _ in range(3)]
    out = [device.empty(n) for _ in range(3)]
    made = expressions(*(x.expression() for x in arrays))

    def seconds(name):
        chunk = C.record_reduce(made[name])
        slots, value, best = (ctypes.c_void_p * 3)(*[g.pointer for g in out]), ctypes.c_double(), 1e9
        for _ in range(8):
            start = time.perf_counter()
            check(lib.sci_cuda_gradient(device.handle, ctypes.byref(chunk), n, 1.0, slots, ctypes.byref(value), 0), device.handle)
            best = min(best, time.perf_counter() - start)
            device.jit_wait()
        return best

    assert seconds("trig") <= 3.5 * seconds("short")  # 2.0 as measured
