"""The limit up to which a tile's digits hold what a product needs (gemm_split.cu, guard_kernel):
sum |a b| >= 0.0021 sqrt(K) in units of the row's and the column's scale. Operands on either side of it,
told apart by their bits: below, the chain of K FMAs; above, one rounding of the sum."""
import math
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
K = 64


def _operands(rng, m, n, both):
    """`both` of the k have both entries at 2^-5 of their scale, every other k one of them (one of those
    the row's or column's largest, against a small entry), so the sum is both 2^-10 and a little."""
    alone = (K - both) // 2
    order = rng.permutation(K)
    shared, ka, kb = order[:both], order[both:both + alone], order[both + alone:]
    a, b = np.full((m, K), 2.0 ** -22), np.full((K, n), 2.0 ** -22)
    a[:, shared] = a[:, ka] = b[shared] = b[kb] = 2.0 ** -5
    a[:, ka[0]], b[kb[0]] = 0.75, 0.75
    return a * (1 + rng.random(a.shape) * 2.0 ** -9), b * (1 + rng.random(b.shape) * 2.0 ** -9)


def _chain(a, b):
    s = Fraction(0)
    for x, y in zip(a, b):
        s = Fraction(float(s + Fraction(x) * Fraction(y)))
    return float(s)


@pytest.mark.parametrize("both,digits", [(12, False), (16, False), (17, False), (18, True), (24, True)])
def test_either_side(lagpu, ctx_fast, both, digits):
    """0.0021 sqrt(64) 2^10 = 17.2. One rounding is half a last place, and the digits left out are below a
    quarter of one here (2^-61 of the scale against 2^-59); the chains are off by more in most elements."""
    torch = pytest.importorskip("torch")
    m, n = 3, 17
    a, b = _operands(np.random.default_rng(both), m, n, both)
    ta, tb = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    tc = torch.zeros((m, n), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    lagpu.matrix_mul_device(ctx_fast, ta.data_ptr(), K, tb.data_ptr(), n, tc.data_ptr(), n, m, K, n)
    ctx_fast.synchronize()
    c = tc.cpu().numpy()
    chain = np.array([[_chain(a[i], b[:, j]) for j in range(n)] for i in range(m)])

    def rounded_once(x):
        out = np.zeros((m, n), dtype=bool)
        for i in range(m):
            for j in range(n):
                e = sum(Fraction(float(p)) * Fraction(float(q)) for p, q in zip(a[i], b[:, j]))
                out[i, j] = abs(Fraction(float(x[i, j])) - e) <= Fraction(math.ulp(float(e))) * 3 / 4
        return out

    assert not rounded_once(chain).all()  # the two can be told apart
    if digits:
        assert rounded_once(c).all()
    else:
        assert np.array_equal(c, chain)
