"""Blocked solves of many right-hand sides and blocked inverses (wavefront blocks of up to 256 rows, split
products between them) against the block-step schedule, at the sizes where the rule begins and where
blocks and tiles do not divide."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


@pytest.mark.parametrize("n,nrhs", [(512, 977), (513, 975), (640, 1001), (1000, 500), (1000, 503),
                                    (1025, 488), (2049, 245), (7813, 64)])
def test_solve_against_block_steps(lagpu, ctx_fast, n, nrhs):
    """Both solve the same factors: backward errors within n u, solutions within their sum times the
    condition of the factors, taken as 1e4 for random matrices of these orders (a few hundred as a rule)."""
    rng = np.random.default_rng(n + nrhs)
    a = rng.standard_normal((n, n)) + 2 * np.sqrt(n) * np.eye(n)[rng.permutation(n)]
    b = rng.standard_normal((n, nrhs))
    lu = lagpu.LUDecomposition.new(a, ctx_fast)
    x = lu.solve(lagpu.Matrix(b, ctx_fast)).data
    ctx_fast.set_option(lagpu.OPT_SOLVE_WAVE, 0)
    y = lu.solve(lagpu.Matrix(b, ctx_fast)).data
    ctx_fast.set_option(lagpu.OPT_SOLVE_WAVE, 2)
    lu.free()
    norm = np.abs(a).sum(axis=1).max()
    for z in (x, y):
        assert (np.abs(a @ z - b).max(axis=0) <= n * U * (norm * np.abs(z).max(axis=0) + 1)).all()
    assert (np.abs(x - y).max(axis=0) <= 2 * n * U * 1e4 * np.abs(y).max(axis=0)).all()


@pytest.mark.parametrize("n", [671, 672, 673, 700, 767, 769, 1025])
@pytest.mark.parametrize("kind", ["random", "graded"])
def test_inverse(lagpu, ctx_fast, n, kind):
    """A X = I column by column: |A X - I| <= n u |A| |X| normwise (growth of partial pivoting on random
    matrices included in the n). Graded: rows and columns over 24 powers of ten, where the products take
    the FMA chains; the bound is taken row by row, as |A| |X| is there."""
    rng = np.random.default_rng(n)
    a = rng.standard_normal((n, n))
    if kind == "graded":
        a = a * 10.0 ** rng.uniform(-6, 6, (n, 1)) * 10.0 ** rng.uniform(-6, 6, (1, n))
    x = lagpu.Matrix(a, ctx_fast).inverse().data
    r = np.abs(a @ x - np.eye(n))
    bound = np.abs(a).sum(axis=1).max() * np.abs(x).max(axis=0)
    assert (r.max(axis=0) <= n * U * bound).all()


def test_inverse_singular(lagpu, ctx_fast):
    a = np.random.default_rng(1).standard_normal((700, 700))
    a[:, 300] = 0.0
    assert lagpu.Matrix(a, ctx_fast).inverse() is None
