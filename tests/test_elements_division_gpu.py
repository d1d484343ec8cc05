"""Integer division, sums and extremes on the device against Python's integers: every pair of bytes, the
magnitudes where the floating-point routes are tightest (multiples and their neighbours, the ends of
the types, 2^52 for 64 bits), zero divisors, and reductions at the edges of a thread's lanes.
"""
import numpy as np
import pytest

from libsci_b200 import chunk as C

pytestmark = pytest.mark.gpu

TYPES = [np.int8, np.uint8, np.int16, np.uint16, np.int32, np.uint32, np.int64, np.uint64]


def truncated(a, b, dtype):
    """C division, 0 for a zero divisor, wrapping for MIN / -1."""
    bits = np.dtype(dtype).itemsize * 8
    out = np.zeros(a.size, dtype)
    for i, (x, y) in enumerate(zip(a.tolist(), b.tolist())):
        q = 0 if y == 0 else abs(x) // abs(y) * (1 if (x < 0) == (y < 0) else -1)
        q &= (1 << bits) - 1
        out[i] = q - (1 << bits) if np.dtype(dtype).kind == "i" and q >> (bits - 1) else q
    return out


def divide(device, a, b):
    da, db = device.array(a), device.array(b)
    return device.evaluate(da.expression() / db.expression()).numpy()


@pytest.mark.parametrize("dtype", [np.int8, np.uint8])
def test_every_byte_pair(device, dtype):
    values = np.arange(256).astype(dtype)
    a, b = np.repeat(values, 256), np.tile(values, 256)
    assert np.array_equal(divide(device, a, b), truncated(a, b, dtype))


@pytest.mark.parametrize("dtype", TYPES)
def test_quotients(device, dtype):
    info, rng = np.iinfo(dtype), np.random.default_rng(5)
    span = [0, 1, 2, 3, info.max, info.max - 1, info.max // 2, info.min, info.min + 1] + [v for p in (7, 15, 16, 22, 23, 31, 32, 51, 52, 53, 62)
                                                                                 for v in (2 ** p - 1, 2 ** p, 2 ** p + 1) if v <= info.max]
    span += [-v for v in span if info.min <= -v < 0]
    edge = np.array([v for v in span if info.min <= v <= info.max], dtype)
    a, b = [np.repeat(edge, edge.size)], [np.tile(edge, edge.size)]
    for bits in range(1, info.bits, max(1, info.bits // 16)):  # multiples of b and their neighbours, of every size
        y = rng.integers(1, min(info.max, 2 ** bits), 2000, dtype=np.uint64, endpoint=True).astype(object)
        k = np.array([int(rng.integers(0, max(1, info.max // int(v)), dtype=np.uint64, endpoint=True)) for v in y], object)
        for off in (-1, 0, 1):
            x = np.array([min(max(int(p) * int(q) + off, 0), info.max) for p, q in zip(y, k)], object)
            sign = rng.integers(0, 2, 2000) * 2 - 1 if info.min < 0 else np.ones(2000, int)
            a.append((x * sign).astype(dtype))
            b.append(y.astype(dtype))
    a, b = np.concatenate(a), np.concatenate(b)
    assert np.array_equal(divide(device, a, b), truncated(a, b, dtype))


@pytest.mark.parametrize("dtype", TYPES)
@pytest.mark.parametrize("count", [1, 3, 8, 17, 4095, 4096, 4097, 100003, 1 << 21])
def test_reductions(device, dtype, count):
    info, rng = np.iinfo(dtype), np.random.default_rng(count)
    x = rng.integers(info.min, info.max, count, dtype=dtype, endpoint=True)
    y = rng.integers(info.min, info.max, count, dtype=dtype, endpoint=True)
    dx, dy = device.array(x), device.array(y)
    plain, product = C.record_reduce(dx.expression()), C.record_reduce(dx.expression() * dy.expression())
    with np.errstate(over="ignore"):
        wrapped = (x * y).astype(dtype)
        assert device.reduce_elements(dtype, product, C.SUM, count) == wrapped.sum(dtype=dtype)
        assert device.reduce_elements(dtype, plain, C.SUM, count) == x.sum(dtype=dtype)
    assert device.reduce_elements(dtype, plain, C.MINIMUM, count) == x.min()
    assert device.reduce_elements(dtype, plain, C.MAXIMUM, count) == x.max()
    assert device.reduce_elements(dtype, product, C.MAXIMUM, count) == wrapped.max()
