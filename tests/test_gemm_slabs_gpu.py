"""Products in slabs of K: the split product takes up to 2^20 terms at a time and adds the rest (C += A B)."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


@pytest.mark.parametrize("m,k,n", [(2, (1 << 20) + 160, 17), (3, 2 * (1 << 20) + 33, 18)])
def test_more_terms_than_one_slab(lagpu, ctx_fast, m, k, n):
    """Positive terms, exact in 53 bits: a slab is rounded once and added once, with an error of its digits
    below its roundings', so 8 u of the sum for up to three slabs. A chain of K FMAs is off by about
    u sqrt(K / 12), 295 u and more."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(k)
    a = rng.integers(1 << 25, 1 << 26, (m, k)).astype(float) * 2.0 ** -26
    b = rng.integers(1 << 25, 1 << 26, (k, n)).astype(float) * 2.0 ** -26
    ta, tb = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    c = torch.zeros((m, n), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    lagpu.matrix_mul_device(ctx_fast, ta.data_ptr(), k, tb.data_ptr(), n, c.data_ptr(), n, m, k, n)
    ctx_fast.synchronize()
    c = c.cpu().numpy()
    for i, j in ((0, 0), (m - 1, n - 1), (0, 9), (m - 1, 3)):
        want = math.fsum(a[i] * b[:, j])
        assert abs(c[i, j] - want) <= 8 * U * want
