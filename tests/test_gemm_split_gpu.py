"""FP64 products on the tensor cores (gemm_split.cu) through la_matrix_mul_device, against the
oracle's Mul (src/matrix/mod.rs:957-980).

Tolerance: the oracle's sum of K rounded products is within (K + 1) u sum |a b| of the exact value
(u = 2^-53), and the split product, rounded once and with digits left out only where they are below
an FMA chain's own error, is held to the same; the two may differ by 2 (K + 1) u sum |a b|."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu
U = 2.0 ** -53

# Edges of the 128 x 64 tiles, of the 32-deep stages and of the 128-deep exact sums, and of the
# rule that takes a product to this path (K >= 32, N > 16).
SHAPES = [(1, 32, 17), (127, 32, 63), (128, 32, 64), (129, 33, 65), (128, 128, 64), (200, 129, 66),
          (257, 160, 130), (64, 513, 40), (130, 1025, 70), (1030, 64, 600)]


def _mul(lagpu, ctx, a, b, ldc=None):
    torch = pytest.importorskip("torch")
    m, k = a.shape
    n = b.shape[1]
    ldc = ldc or n
    ta, tb = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    tc = torch.full((m, ldc), 7.0, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    lagpu.matrix_mul_device(ctx, ta.data_ptr(), k, tb.data_ptr(), n, tc.data_ptr(), ldc, m, k, n)
    ctx.synchronize()
    c = tc.cpu().numpy()
    assert np.all(c[:, n:] == 7.0)  # nothing is written beside the product
    return c[:, :n]


def _close(c, a, b):
    k = a.shape[1]
    ref = oracle.matmul(a, b)
    with np.errstate(over="ignore"):
        lim = 2 * (k + 1) * U * (np.abs(a) @ np.abs(b))
    assert np.all(np.abs(c - ref) <= lim)


@pytest.mark.parametrize("mkn", SHAPES)
def test_gaussian(lagpu, ctx_fast, mkn):
    m, k, n = mkn
    rng = np.random.default_rng(m * 31 + k * 7 + n)
    a, b = rng.standard_normal((m, k)), rng.standard_normal((k, n))
    _close(_mul(lagpu, ctx_fast, a, b, n + 3), a, b)


@pytest.mark.parametrize("mkn", SHAPES[3:8])
def test_whole_numbers_are_exact(lagpu, ctx_fast, mkn):
    m, k, n = mkn
    rng = np.random.default_rng(m + k + n)
    a = rng.integers(-1000, 1001, (m, k)).astype(float)
    b = rng.integers(-1000, 1001, (k, n)).astype(float)
    assert np.array_equal(_mul(lagpu, ctx_fast, a, b), oracle.matmul(a, b))


@pytest.mark.parametrize("kind", ["rowscale", "beyond", "outlier", "graded", "sparse", "zero",
                                  "denormal", "constant"])
def test_ranges(lagpu, ctx_fast, kind):
    # Rows and columns of very different size stay on the tensor cores; outliers, graded and sparse
    # operands and exponents beyond the digits' range take the FMA tiles, some tiles of a product or
    # all.
    m, k, n = 300, 200, 140
    rng = np.random.default_rng(len(kind))
    a, b = rng.standard_normal((m, k)), rng.standard_normal((k, n))
    if kind == "rowscale":
        a *= np.exp2(rng.integers(-390, 391, (m, 1)))
        b *= np.exp2(rng.integers(-20, 21, (1, n)))
    elif kind == "beyond":
        a[::50] *= 2.0 ** 450
        a[1::50] *= 2.0 ** -450
    elif kind == "outlier":
        a[5, 7] = 1e9
        b[3, 100] = -1e12
    elif kind == "graded":
        s = np.logspace(-8, 8, k)
        a, b = a * s, b / s[:, None]
    elif kind == "sparse":
        a *= rng.random((m, k)) < 0.1
    elif kind == "zero":
        a[:150] = 0.0
        b[:, 64:128] = 0.0
    elif kind == "denormal":
        a[10] = 5e-324 * rng.integers(0, 100, k)
        a[20, ::2] = 1e-310
    else:
        a[:], b[:] = 1.0 / 3.0, -2.0 / 3.0
    c = _mul(lagpu, ctx_fast, a, b)
    _close(c, a, b)
    if kind == "zero":
        assert np.all(c[:150] == 0.0) and np.all(c[:, 64:128] == 0.0)


def test_values_that_are_not_finite(lagpu, ctx_fast):
    m, k, n = 260, 96, 130
    rng = np.random.default_rng(3)
    a, b = rng.standard_normal((m, k)), rng.standard_normal((k, n))
    a[3, 5], a[140, 6], b[9, 70], b[11, 10] = np.nan, np.inf, -np.inf, np.nan
    c, ref = _mul(lagpu, ctx_fast, a, b), oracle.matmul(a, b)
    assert np.array_equal(np.isnan(c), np.isnan(ref))
    inf = np.isinf(ref)
    assert np.array_equal(c[inf], ref[inf])
    ok = np.isfinite(ref)
    a0, b0 = np.where(np.isfinite(a), a, 0), np.where(np.isfinite(b), b, 0)
    assert np.all(np.abs(c - ref)[ok] <= (2 * (k + 1) * U * (np.abs(a0) @ np.abs(b0)))[ok])


def test_update_form(lagpu, ctx_fast):
    # C -= A B, which the factorization runs with K = 64: L U against P A.
    rng = np.random.default_rng(8)
    a = rng.standard_normal((321, 321))
    ref = oracle.lu_factor(a)
    lu = lagpu.LUDecomposition.new(a, ctx_fast)
    assert np.array_equal(lu.get_piv(), ref.piv)
    l, u = lu.get_l().data, lu.get_u().data
    pa = a[ref.piv.astype(int)]
    assert np.all(np.abs(l @ u - pa) <= 2 * 323 * U * (np.abs(l) @ np.abs(u)))
