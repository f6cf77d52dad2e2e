"""Which schedule a solve of many right-hand sides takes (lu_solve_inplace): blocks with split products
between them; where U's rows lie unevenly, so that the products' tiles are FMA chains, only from
n nrhs = 800000 on instead of 500000."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def _matrix(kind, n):
    rng = np.random.default_rng(n + len(kind))
    a = rng.standard_normal((n, n))
    i, j = np.arange(n)[:, None], np.arange(n)
    if kind == "banded":
        return a * (np.abs(i - j) <= 8) + 20.0 * (i == j)
    if kind == "columns":
        return a * np.logspace(-8, 8, n)
    if kind == "columns back":
        return a * np.logspace(8, -8, n)
    if kind == "dominant":
        return a + 2 * np.sqrt(n) * np.eye(n)[rng.permutation(n)]
    return a * np.logspace(-8, 8, n)[rng.permutation(n)][:, None] if kind == "rows" else a


@pytest.mark.parametrize("n,nrhs", [(512, 1000), (1000, 500), (2500, 256), (1000, 801)])
@pytest.mark.parametrize("kind,blocked", [("random", True), ("dominant", True), ("rows", True),
                                          ("banded", False), ("columns", False), ("columns back", False)])
def test_schedule_and_backward_error(lagpu, ctx_fast, kind, blocked, n, nrhs):
    """The wavefront is a permutation and two launches. Backward error row by row: |A X - B| <= 3 n u
    |L| |U| |X| (Higham, Accuracy and Stability of Numerical Algorithms, theorem 9.4)."""
    a = _matrix(kind, n)
    b = np.random.default_rng(nrhs).standard_normal((n, nrhs))
    lu = lagpu.LUDecomposition.new(a, ctx_fast)
    before = ctx_fast.kernel_launches()
    x = lu.solve(lagpu.Matrix(b, ctx_fast)).data
    launches = ctx_fast.kernel_launches() - before
    p, l, u = lu.get_piv().astype(int), lu.get_l().data, lu.get_u().data
    lu.free()
    assert (launches > 3) == (blocked or n * nrhs >= 800000)
    bound = 3 * n * U * (np.abs(l) @ (np.abs(u) @ np.abs(x)))
    assert np.all(np.abs(a @ x - b)[p] <= bound)
