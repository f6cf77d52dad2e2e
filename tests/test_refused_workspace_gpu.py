"""Memory that a call can do without (the digits of the split products, the staging of host copies) is
refused, allocation by allocation: the call then returns LA_OK with an answer as exact as any and leaves no
error text, or LA_NOMEM with one. The forms without digits are FMA products throughout."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def _lu(lagpu, ctx, a):
    lu = lagpu.LUDecomposition.new(a, ctx)
    p, l, u = lu.get_piv().astype(int), lu.get_l().data, lu.get_u().data
    lu.free()
    # Higham, Accuracy and Stability of Numerical Algorithms, theorem 9.3, twice
    return np.all(np.abs(l @ u - a[p]) <= 2 * (len(a) + 2) * U * (np.abs(l) @ np.abs(u)))


def _chol(lagpu, ctx, a):
    n = len(a)
    s = a @ a.T / n + 0.1 * np.eye(n)
    s = np.tril(s) + np.tril(s, -1).T
    c = lagpu.CholeskyDecomposition.new(s, ctx)
    l = c.get_l().data
    c.free()
    return np.all(np.abs(l @ l.T - s) <= 2 * (n + 2) * U * (np.abs(l) @ np.abs(l).T))  # theorem 10.3


def _qr(lagpu, ctx, a):
    n = len(a)
    qr = lagpu.QRDecomposition.new(a, ctx)
    q, r = qr.get_q().data, qr.get_r().data
    qr.free()
    return (np.all(np.linalg.norm(q @ r - a, axis=0) <= 16 * n * U * np.linalg.norm(a, axis=0)) and
            np.linalg.norm(q.T @ q - np.eye(n), axis=0).max() <= 16 * n * U)  # theorem 19.4


def _mul(lagpu, ctx, a):
    n = len(a)
    c = (lagpu.Matrix(a, ctx) * lagpu.Matrix(a.T.copy(), ctx)).data
    return np.all(np.abs(c - a @ a.T) <= 2 * (n + 1) * U * (np.abs(a) @ np.abs(a).T))


def _solve(lagpu, ctx, a):
    n = len(a)
    b = np.random.default_rng(2).standard_normal((n, 901))
    lu = lagpu.LUDecomposition.new(a, ctx)
    x = lu.solve(lagpu.Matrix(b, ctx)).data
    l, u, p = lu.get_l().data, lu.get_u().data, lu.get_piv().astype(int)
    lu.free()
    return np.all(np.abs(a @ x - b)[p] <= 3 * n * U * (np.abs(l) @ (np.abs(u) @ np.abs(x))))  # theorem 9.4


def _inverse(lagpu, ctx, a):
    x = lagpu.Matrix(a, ctx).inverse().data
    bound = np.abs(a).sum(axis=1).max() * np.abs(x).max(axis=0)
    return np.all(np.abs(a @ x - np.eye(len(a))).max(axis=0) <= len(a) * U * bound)


@pytest.mark.parametrize("call,n,allocations", [(_lu, 301, 5), (_lu, 700, 4), (_chol, 303, 4), (_chol, 800, 3),
                                                (_qr, 301, 11), (_mul, 201, 5), (_solve, 701, 9),
                                                (_inverse, 701, 7)])
def test_allocation_by_allocation(lagpu, call, n, allocations):
    a = np.random.default_rng(n).standard_normal((n, n))
    done = 0
    for k in range(1, allocations + 1):
        ctx = lagpu.Context(0, lagpu.ARITH_FAST)
        try:
            ctx.set_option(lagpu.OPT_INJECT_ALLOC_FAIL, k)
            try:
                assert call(lagpu, ctx, a)
                assert ctx.last_error() == ""
                done += 1
            except lagpu.LaError as e:
                assert e.status == lagpu.NOMEM and "injected" in ctx.last_error()
            assert ctx.get_option(lagpu.OPT_INJECT_ALLOC_FAIL) == 0  # there was a k-th allocation
        finally:
            ctx.close()
    assert done >= 1  # one of them at least is the digits'
