"""Host calls whose result goes where an argument came from: the argument is on its way to the device until the
stream has taken it, so nothing may change it before."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _p(a):
    return ctypes.c_void_p(a.ctypes.data)


@pytest.mark.parametrize("n,nrhs", [(33, 3), (700, 5), (2501, 33), (1001, 1001)])
def test_lu_solve(lagpu, ctx_fast, n, nrhs):
    rng = np.random.default_rng(n)
    lu = lagpu.LUDecomposition.new(rng.standard_normal((n, n)), ctx_fast)
    b = rng.standard_normal((n, nrhs))
    x = np.empty_like(b)
    solve = lagpu.lib().la_lu_solve
    for _ in range(5):
        y = b.copy()
        assert solve(lu.h, _p(b), n, nrhs, _p(x)) == lagpu.OK
        assert solve(lu.h, _p(y), n, nrhs, _p(y)) == lagpu.OK
        assert np.array_equal(x, y)
    lu.free()


@pytest.mark.parametrize("n", [33, 701, 2501])
def test_mul(lagpu, ctx_fast, n):
    rng = np.random.default_rng(n)
    a, b = rng.standard_normal((n, n)), rng.standard_normal((n, n))
    c = np.empty_like(a)
    mul = lagpu.lib().la_matrix_mul
    for _ in range(3):
        left, right = a.copy(), b.copy()
        assert mul(ctx_fast.h, _p(a), n, n, _p(b), n, n, _p(c)) == lagpu.OK
        assert mul(ctx_fast.h, _p(left), n, n, _p(b), n, n, _p(left)) == lagpu.OK
        assert mul(ctx_fast.h, _p(a), n, n, _p(right), n, n, _p(right)) == lagpu.OK
        assert np.array_equal(left, c) and np.array_equal(right, c)


@pytest.mark.parametrize("n", [130, 701])
def test_inverse_and_qr(lagpu, ctx_fast, n):
    rng = np.random.default_rng(n)
    a = rng.standard_normal((n, n))
    out, same = np.empty_like(a), a.copy()
    inv = lagpu.lib().la_matrix_inverse
    assert inv(ctx_fast.h, _p(a), n, n, _p(out)) == lagpu.OK and inv(ctx_fast.h, _p(same), n, n, _p(same)) == lagpu.OK
    assert np.array_equal(out, same)
    qr = lagpu.QRDecomposition.new(a, ctx_fast)
    b = rng.standard_normal((n, 3))
    x, y = np.empty_like(b), b.copy()
    solve = lagpu.lib().la_qr_solve
    assert solve(qr.h, _p(b), n, 3, _p(x)) == lagpu.OK and solve(qr.h, _p(y), n, 3, _p(y)) == lagpu.OK
    qr.free()
    assert np.array_equal(x, y)
