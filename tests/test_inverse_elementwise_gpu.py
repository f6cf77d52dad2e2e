"""Inverses of matrices whose rows and columns differ by many powers of ten, element by element: a bound by
norms would only see the largest rows and columns."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def _ratio(a, x, l, u, p):
    """max |A X - I| / (|P'L| |U| |X|): two triangular solves per column give 3 n u of it (Higham, Accuracy
    and Stability of Numerical Algorithms, theorem 9.4), the product here another n u."""
    lu = np.empty_like(a)
    lu[p] = np.abs(l) @ np.abs(u)
    return (np.abs(a @ x - np.eye(len(a))) / (lu @ np.abs(x))).max()


@pytest.mark.parametrize("n", [64, 130, 671, 672, 673, 769, 1025])
@pytest.mark.parametrize("kind", ["random", "graded", "banded"])
def test_inverse(lagpu, ctx_fast, n, kind):
    rng = np.random.default_rng(n)
    a = rng.standard_normal((n, n))
    if kind == "graded":
        a = a * 10.0 ** rng.uniform(-6, 6, (n, 1)) * 10.0 ** rng.uniform(-6, 6, (1, n))
    elif kind == "banded":
        i, j = np.arange(n)[:, None], np.arange(n)
        a = (a * (np.abs(i - j) <= 6) + 8.0 * (i == j)) * 10.0 ** rng.uniform(-6, 6, (n, 1))
    lu = lagpu.LUDecomposition.new(a, ctx_fast)
    l, u, p = lu.get_l().data, lu.get_u().data, lu.get_piv().astype(int)
    lu.free()
    x = lagpu.Matrix(a, ctx_fast).inverse().data
    assert _ratio(a, x, l, u, p) <= 4 * n * U
    wrong = x * (1 + 1e-9 * rng.standard_normal(x.shape))
    assert _ratio(a, wrong, l, u, p) > 4 * n * U
