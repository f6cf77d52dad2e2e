"""QR of matrices whose blocks' products leave most tiles to FMA chains (entries over many powers of ten, a
band): after such a product the next ones form no digits (gemm_split.cu, skips_digits)."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def _skew(rng, m, n):
    return rng.standard_normal((m, n)) * np.exp(4 * rng.standard_normal((m, n)))


def _matrix(kind, m, n):
    """mixed: the first half of the columns and rows skewed, the rest even, so that products of both kinds
    follow each other, in both directions over get_q."""
    rng = np.random.default_rng(m + n)
    a = _skew(rng, m, n)
    if kind == "mixed":
        a[m // 2:] = rng.standard_normal((m - m // 2, n))
        a[:, n // 2:] = rng.standard_normal((m, n - n // 2)) * 100
    elif kind == "banded":
        a = a * (np.abs(np.arange(m)[:, None] - np.arange(n)) <= 6)
        a[np.arange(n), np.arange(n)] += 12
    return a


@pytest.mark.parametrize("kind", ["skew", "mixed", "banded"])
@pytest.mark.parametrize("m,n", [(260, 130), (700, 700), (1100, 1001), (900, 1300)])
def test_factors(lagpu, ctx_fast, kind, m, n):
    """Column by column, |A - Q R| <= 16 r u |a_j| in the 2-norm and Q'Q = I within 16 r u: r = min(m, n)
    reflections with a few u of their own each (Higham, Accuracy and Stability of Numerical Algorithms,
    theorem 19.4)."""
    a = _matrix(kind, m, n) if kind != "banded" or m >= n else _matrix(kind, n, m).T.copy()
    qr = lagpu.QRDecomposition.new(a, ctx_fast)
    q, r = qr.get_q().data, qr.get_r().data
    qr.free()
    k = min(m, n)
    assert np.all(np.linalg.norm(q @ r - a, axis=0) <= 16 * k * U * np.linalg.norm(a, axis=0))
    q = q[:, :k]
    assert np.linalg.norm(q.T @ q - np.eye(k), axis=0).max() <= 16 * k * U


def test_no_slower_than_without_digits(lagpu, ctx_fast):
    """Within 8 % of the same factorization where the digits get no memory (1.12 when every block formed
    and rejected its digits, 1.05 now)."""
    torch = pytest.importorskip("torch")
    m, n = 2500, 1501
    a = torch.from_numpy(_matrix("skew", m, n)).cuda()
    torch.cuda.synchronize()

    def seconds(refuse):
        ctx_fast.set_option(lagpu.OPT_INJECT_ALLOC_FAIL, refuse)
        t = time.perf_counter()
        try:
            qr = lagpu.QRDecomposition.new_device(a.data_ptr(), n, m, n, ctx_fast)
        except lagpu.LaError:
            return None
        finally:
            ctx_fast.set_option(lagpu.OPT_INJECT_ALLOC_FAIL, 0)
        ctx_fast.synchronize()
        t = time.perf_counter() - t
        qr.free()
        return t

    seconds(0)
    digits = next(k for k in range(1, 12) if seconds(k) is not None)  # the one that can be done without
    pairs = [(seconds(0), seconds(digits)) for _ in range(10)]
    assert min(p[0] for p in pairs) <= 1.08 * min(p[1] for p in pairs)
