"""Products whose tiles the digits do not hold (gemm_split.cu, fma_pieces): graded, banded, triangular and
sparse operands, whose tiles are FMA chains in pieces of 64, 32 or 16 rows and 16 columns.

Such a product is the same chain of FMAs per element, in ascending k, that the FMA kernels perform where
the digits get no memory (refused here by LA_OPT_INJECT_ALLOC_FAIL): the same bits, and no slower."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def _graded(m, k, n, seed=0):
    """Along k: a tile's products are all of one size, its digits hold none of the small operands."""
    rng = np.random.default_rng(seed + m + k + n)
    s = np.logspace(-30, 30, k)
    return rng.standard_normal((m, k)) * s, rng.standard_normal((k, n)) / s[:, None]


class _Mul:
    def __init__(self, lagpu, ctx, a, b):
        torch = pytest.importorskip("torch")
        self.lagpu, self.ctx = lagpu, ctx
        self.m, self.k, self.n = a.shape[0], a.shape[1], b.shape[1]
        self.a, self.b = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
        self.c = torch.zeros((self.m, self.n), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()

    def __call__(self, refuse):
        """Seconds; the product is in c. refuse: the digits get no memory."""
        if refuse:
            self.ctx.set_option(self.lagpu.OPT_INJECT_ALLOC_FAIL, 1)
        t = time.perf_counter()
        self.lagpu.matrix_mul_device(self.ctx, self.a.data_ptr(), self.k, self.b.data_ptr(), self.n,
                                     self.c.data_ptr(), self.n, self.m, self.k, self.n)
        self.ctx.synchronize()
        t = time.perf_counter() - t
        assert self.ctx.get_option(self.lagpu.OPT_INJECT_ALLOC_FAIL) == 0
        return t


# Few pieces (16 rows each), some (32) and many (64); one row or column of tiles, remainders of every
# piece and slab.
@pytest.mark.parametrize("mkn", [(1, 32, 17), (15, 33, 18), (16, 32, 32), (17, 31 + 32, 33), (64, 64, 64),
                                 (65, 95, 49), (129, 100, 66), (100, 1000, 257), (513, 65, 390),
                                 (1025, 70, 1030)])
def test_same_bits_as_the_fma_kernels(lagpu, ctx_fast, mkn):
    mul = _Mul(lagpu, ctx_fast, *_graded(*mkn))
    mul(False)
    c = mul.c.cpu().numpy()
    mul(True)
    assert np.array_equal(c, mul.c.cpu().numpy())


@pytest.mark.parametrize("mkn", [(100, 64, 100), (300, 200, 140), (64, 2048, 2048), (64, 1936, 436),
                                 (1000, 1000, 1000)])
def test_no_slower_than_the_fma_kernels(lagpu, ctx_fast, mkn):
    """Within 10 % of the kernels that would run without digits (1.08 to 1.33 times as long when a piece
    was 64 x 64 and a padded half of a tile a piece like any other)."""
    mul = _Mul(lagpu, ctx_fast, *_graded(*mkn))
    mul(False), mul(True)
    pairs = [(mul(False), mul(True)) for _ in range(30)]
    assert min(p[0] for p in pairs) <= 1.1 * min(p[1] for p in pairs)


def _operand(kind, m, n):
    rng = np.random.default_rng(m + 3 * n)
    a = rng.standard_normal((m, n))
    i, j = np.arange(m)[:, None], np.arange(n)
    if kind == "graded":
        return a * np.logspace(-8, 8, m)[:, None] * np.logspace(6, -6, n)
    if kind == "banded":
        return a * (np.abs(i - j) <= 6) + 12.0 * (i == j)
    if kind == "triangular":
        return a * (i <= j) + 8.0 * (i == j)
    return a * (rng.random((m, n)) < 0.02) + (i == j)


KINDS = ["graded", "banded", "triangular", "sparse"]


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("m,n", [(333, 333), (700, 520), (1100, 1100)])
def test_lu(lagpu, ctx_fast, kind, m, n):
    """|P A - L U| <= 2 (n + 2) u |L| |U| element by element: every element is one sum of at most n terms
    and a quotient (Higham, Accuracy and Stability of Numerical Algorithms, theorem 9.3), twice that, and
    the check's own product."""
    a = _operand(kind, m, n)
    lu = lagpu.LUDecomposition.new(a, ctx_fast)
    p, l, u = lu.get_piv().astype(int), lu.get_l().data, lu.get_u().data
    lu.free()
    l, u = l[:, :n], u[:n]
    assert np.all(np.abs(l @ u - a[p]) <= 2 * (n + 2) * U * (np.abs(l) @ np.abs(u)))


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("m,n", [(333, 333), (900, 450), (450, 700)])
def test_qr(lagpu, ctx_fast, kind, m, n):
    """Column by column, |A - Q R| <= 16 r u |a_j| in the 2-norm and Q'Q = I within 16 r u: r = min(m, n)
    reflections with a few u of their own each (theorem 19.4 there)."""
    a = _operand(kind, m, n)
    qr = lagpu.QRDecomposition.new(a, ctx_fast)
    q, r = qr.get_q().data, qr.get_r().data
    qr.free()
    k = min(m, n)
    assert np.all(np.linalg.norm(q @ r - a, axis=0) <= 16 * k * U * np.linalg.norm(a, axis=0))
    q = q[:, :k]
    assert np.linalg.norm(q.T @ q - np.eye(k), axis=0).max() <= 16 * k * U


@pytest.mark.parametrize("kind", ["graded", "banded", "diagonal"])
@pytest.mark.parametrize("n", [333, 800, 1100])
def test_cholesky(lagpu, ctx_fast, kind, n):
    """|L L' - A| <= 2 (n + 2) u |L| |L'| element by element (theorem 10.3 there, twice that)."""
    rng = np.random.default_rng(n)
    i, j = np.arange(n)[:, None], np.arange(n)
    if kind == "graded":
        g, s = rng.standard_normal((n, n + 3)), np.logspace(-8, 8, n)[rng.permutation(n)]
        a = (g @ g.T / n + 0.1 * np.eye(n)) * s[:, None] * s
        a = np.tril(a) + np.tril(a, -1).T
    elif kind == "banded":
        a = 2.0 * (i == j) - 1.0 * (np.abs(i - j) == 1)
    else:
        a = (i == j) * np.logspace(-20, 20, n)
    c = lagpu.CholeskyDecomposition.new(a, ctx_fast)
    assert c is not None
    l = c.get_l().data
    c.free()
    assert np.array_equal(l, np.tril(l))
    assert np.all(np.abs(l @ l.T - a) <= 2 * (n + 2) * U * (np.abs(l) @ np.abs(l).T))
