"""The solves' items of 128 rows of one column (up to 24 right-hand sides) against the block-step schedule:
the same bits, at the edges of blocks and items and on both sides of the rule."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _both(lagpu, ctx, a, b):
    lu = lagpu.LUDecomposition.new(a, ctx)
    x = lu.solve(lagpu.Matrix(b, ctx)).data
    ctx.set_option(lagpu.OPT_SOLVE_WAVE, 0)
    y = lu.solve(lagpu.Matrix(b, ctx)).data
    ctx.set_option(lagpu.OPT_SOLVE_WAVE, 2)
    lu.free()
    return x, y


@pytest.mark.parametrize("n", [1, 31, 32, 33, 63, 65, 96, 97, 127, 128, 129, 159, 161, 255, 256, 257, 385, 1000])
@pytest.mark.parametrize("arith", ["fast", "exact"])
def test_same_bits(lagpu, ctx_fast, ctx_exact, n, arith):
    ctx = ctx_fast if arith == "fast" else ctx_exact
    rng = np.random.default_rng(n)
    a = rng.standard_normal((n, n))
    for nrhs in (1, 3, 24, 25):
        x, y = _both(lagpu, ctx, a, rng.standard_normal((n, nrhs)))
        assert np.array_equal(x.view(np.uint64), y.view(np.uint64)), nrhs


@pytest.mark.parametrize("arith", ["fast", "exact"])
def test_not_finite(lagpu, ctx_fast, ctx_exact, arith):
    """Infinities and NaN, the NaN of all ones among them, pass from block to block; nothing waits for them."""
    ctx = ctx_fast if arith == "fast" else ctx_exact
    rng = np.random.default_rng(2)
    n = 300
    a, b = rng.standard_normal((n, n)), rng.standard_normal((n, 4))
    b[7, 0] = np.inf
    b[200, 1] = np.nan
    b.view(np.uint64)[5, 2] = 0xFFFFFFFFFFFFFFFF
    b.view(np.uint64)[299, 2] = 0xFFFFFFFFFFFFFFFF
    with np.errstate(all="ignore"):
        x, y = _both(lagpu, ctx, a, b)
    assert np.array_equal(x, y, equal_nan=True)
    assert np.all(np.isfinite(x[:, 3])) and not np.any(np.isfinite(x[:, 2]))


@pytest.mark.parametrize("n", [97, 129, 300])
def test_cholesky(lagpu, ctx_exact, oracle_lib, n):
    rng = np.random.default_rng(n)
    g = rng.standard_normal((n, n))
    a = g @ g.T + n * np.eye(n)
    a = (a + a.T) * 0.5
    b = rng.standard_normal((n, 2))
    ch = lagpu.CholeskyDecomposition.new(lagpu.Matrix(a, ctx_exact))
    x = ch.solve(lagpu.Matrix(b, ctx_exact)).data
    ch.free()
    assert np.array_equal(x, oracle.chol_solve(oracle.chol_new(a), b))
