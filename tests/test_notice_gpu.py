"""Blocking reductions, whose value the kernel writes to pinned host memory and announces: one block and
many, back to back with queued work, after an empty one, from several contexts and threads.
"""
import threading

import numpy as np
import pytest

from libsci_b200 import chunk as C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 31, 2047, 2048, 2049, 100003, 1 << 22])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_values(device, count, dtype):
    x = (np.arange(count) % 1009 - 500).astype(dtype)  # every partial sum is exact
    d = device.array(x)
    for fold, want in ((C.SUM, x.sum(dtype=np.float64)), (C.MINIMUM, x.min()), (C.MAXIMUM, x.max())):
        chunk = C.record_reduce(d.expression())
        assert device.reduce_chunk(chunk, fold, count) == want
    assert device.reduce_chunk(chunk, C.SUM, 0) == 0.0
    doubled = device.evaluate(d + d)  # queued, then reduced at once
    assert device.reduce_chunk(C.record_reduce(doubled.expression()), C.SUM, count) == 2.0 * x.sum(dtype=np.float64)
    x[count // 2] = np.nan
    d.upload(x)
    assert np.isnan(device.reduce_chunk(chunk, C.MAXIMUM, count))


def test_threads_and_contexts():
    from libsci_b200.device import Device

    shared = Device(0)
    failures = []

    def work(seed, own):
        dev = Device(0) if own else shared
        x = np.random.default_rng(seed).integers(-99, 99, 5000 + seed).astype(np.float32)
        d = dev.array(x)
        chunk = C.record_reduce(d.expression())
        for _ in range(200):
            if dev.reduce_chunk(chunk, C.SUM, x.size) != x.sum(dtype=np.float64):
                failures.append(seed)
        if own:
            dev.close()

    threads = [threading.Thread(target=work, args=(s, s % 2 == 0)) for s in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    shared.close()
    assert not failures
