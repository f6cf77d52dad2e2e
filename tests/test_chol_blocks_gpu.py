"""FAST Cholesky at the edges of its blocks: 32-column panels (32 rows per CTA, then passes of 64),
blocks of 64, 128 and 256 columns, the 128 x 64 tiles of the trailing update.

Tolerance: a Cholesky factor computed in any order satisfies |L L' - A| <= (n + 2) u |L| |L|'
(Higham, Accuracy and Stability of Numerical Algorithms, theorem 10.3, with one more rounding for the
reciprocal square root); twice that."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
U = 2.0 ** -53

SIZES = [1, 2, 31, 32, 33, 63, 64, 65, 95, 96, 97, 128, 129, 161, 256, 257, 400, 768, 769, 833, 2049,
         2307, 5003]


@pytest.mark.parametrize("n", SIZES)
def test_factor(lagpu, ctx_fast, n):
    torch = pytest.importorskip("torch")
    g = np.random.default_rng(n).standard_normal((n, n + 3))
    a = torch.from_numpy(g).cuda()
    a = a @ a.t() / n + 0.1 * torch.eye(n, dtype=torch.float64, device="cuda")
    a = ((a + a.t()) / 2).contiguous()
    torch.cuda.synchronize()
    c = lagpu.CholeskyDecomposition.new_device(a.data_ptr(), n, n, ctx_fast)
    assert c is not None
    l = torch.from_numpy(c.get_l().data).cuda()
    c.free()
    assert torch.equal(l, torch.tril(l))
    lim = 2 * (n + 2) * U * (l.abs() @ l.abs().t())
    assert bool(((l @ l.t() - a).abs() <= lim).all())


@pytest.mark.parametrize("n,k", [(40, 35), (70, 0), (70, 33), (300, 299), (1000, 640)])
def test_not_positive_definite(lagpu, ctx_fast, n, k):
    g = np.random.default_rng(n + k).standard_normal((n, n))
    a = g @ g.T / n + np.eye(n)
    a[k, k] = -1.0
    assert lagpu.CholeskyDecomposition.new((a + a.T) / 2, ctx_fast) is None
