"""Integer chunks whose temporaries change the block's threads (256, 128, 64): stored and reduced, against
numpy's wrapping integers. Counts give one block, every block of a launch and several tiles each."""
import numpy as np
import pytest

from libsci_b200 import chunk as C

pytestmark = pytest.mark.gpu


def wide_chunk(dtype, pointer, temporaries):
    """x + 0, x + 1, ... in temporaries of their own, then the sum of the first and the last."""
    chunk = C._new_chunk(dtype)
    source = chunk.input(pointer)
    made = [chunk.emit(C.CODE["subtract"], source, chunk.constant(float(-k))) for k in range(temporaries)]
    return chunk, chunk.emit(C.CODE["add"], made[0], made[-1])


@pytest.mark.parametrize("dtype", [np.int8, np.int32, np.int64])
@pytest.mark.parametrize("temporaries", [2, 6, 7, 12, 13, 25, 55, 56, 57, 60])
def test_block_sizes(device, dtype, temporaries):
    info, rng = np.iinfo(dtype), np.random.default_rng(temporaries)
    for count in (1, 4097, 3000003):
        x = rng.integers(info.min, info.max, count, dtype=dtype, endpoint=True)
        with np.errstate(over="ignore"):
            want = (x + (x + dtype(temporaries - 1))).astype(dtype)
        dx, out = device.array(x), device.empty(count, dtype)
        chunk, value = wide_chunk(dtype, dx.pointer, temporaries)
        assert device.reduce_elements(dtype, chunk.reduce(value), C.SUM, count) == want.sum(dtype=dtype)
        assert device.reduce_elements(dtype, chunk, C.MINIMUM, count) == want.min()
        device.execute_elements(dtype, chunk.output(value), out.pointer, count)
        assert chunk.valid() and chunk.temporaries >= temporaries and np.array_equal(out.numpy(), want)
