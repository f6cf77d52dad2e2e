"""Results to host memory whose rows are not a multiple of the device pitch: into memory that the process has
touched and into fresh pages, at any offset in a page, and no byte outside the result."""
import ctypes
import mmap
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _factor(lagpu, ctx, n):
    c = lagpu.CholeskyDecomposition.new(np.eye(n) * np.arange(1, n + 1) ** 2.0, ctx)
    return c, np.diag(np.arange(1.0, n + 1))


@pytest.mark.parametrize("n", [1, 2, 3, 91, 181, 333, 1001])
@pytest.mark.parametrize("fresh", [False, True])
@pytest.mark.parametrize("offset", [0, 8, 4088, 65528])
def test_values(lagpu, ctx_fast, n, fresh, offset):
    c, want = _factor(lagpu, ctx_fast, n)
    mm = mmap.mmap(-1, offset + 8 * n * n + 65536)
    b = np.frombuffer(mm, dtype=np.uint8)
    if not fresh:
        b[:] = 0x5a
    assert lagpu.lib().la_chol_get_l(c.h, ctypes.c_void_p(b.ctypes.data + offset)) == lagpu.OK
    c.free()
    rest = 0 if fresh else 0x5a
    assert np.all(b[:offset] == rest) and np.all(b[offset + 8 * n * n:] == rest)
    assert np.array_equal(b[offset:offset + 8 * n * n].view(np.float64).reshape(n, n), want)


def test_padded_no_slower_than_dense(lagpu, ctx_fast):
    """L of order 901 (rows padded to 904 on the device) takes no more than 1.2 times as long as L of order 900, which
    is one contiguous copy (1.27 times through a dense buffer on the device)."""
    a, b = _factor(lagpu, ctx_fast, 901)[0], _factor(lagpu, ctx_fast, 900)[0]
    out = np.ones((901, 901))

    def seconds(c):
        t = time.perf_counter()
        assert lagpu.lib().la_chol_get_l(c.h, ctypes.c_void_p(out.ctypes.data)) == lagpu.OK
        return time.perf_counter() - t

    pairs = [(seconds(a), seconds(b)) for _ in range(100)]
    a.free()
    b.free()
    assert min(p[0] for p in pairs[5:]) <= 1.2 * min(p[1] for p in pairs[5:])
