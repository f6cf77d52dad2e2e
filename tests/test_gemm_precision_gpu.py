"""How exact products by splitting are, where their tiles are not left to FMA chains: half a last place of the
result, and the products of digits that are left out."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _exact(a, b):
    """a b as whole numbers of 2^-e: every entry is a whole number of 2^-60 here, of at most 60 bits."""
    ia = (np.ldexp(a, 60)).astype(np.int64).astype(object)
    ib = (np.ldexp(b, 60)).astype(np.int64).astype(object)
    return ia @ ib


def _scale(x, axis):
    """2^ea with |x| < 2^ea along the axis."""
    return np.exp2(np.frexp(np.abs(x).max(axis=axis))[1])


@pytest.mark.parametrize("mkn", [(40, 32, 17), (33, 64, 40), (64, 100, 33), (48, 256, 48), (20, 700, 30),
                                 (17, 2049, 20)])
@pytest.mark.parametrize("kind", ["normal", "uniform", "positive"])
def test_error(lagpu, ctx_fast, mkn, kind):
    """|c - a b| <= ulp(a b) / 2 + 9.1 K 2^-64 2^(ea + eb): one rounding of the sum; left out per term, with
    digits up to 2^7 in units of 2^-(7 + 8 s), are sum over s + t > 7 of 2^-(8 (s + t)) <= 7.1 * 2^-64, and
    2 * 2^-64 of the values' own last digits. Seven digits would leave out 2^8 times as much."""
    torch = pytest.importorskip("torch")
    m, k, n = mkn
    rng = np.random.default_rng(m + k + n)
    draw = {"normal": lambda s: np.clip(rng.standard_normal(s), -7, 7), "uniform": lambda s: rng.uniform(-1, 1, s),
            "positive": lambda s: rng.uniform(0.5, 1, s)}[kind]
    # whole numbers of 2^-60, below 1
    a, b = (np.ldexp(np.rint(np.ldexp(draw(s) / 8, 60)), -60) for s in ((m, k), (k, n)))
    ta, tb = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    tc = torch.zeros((m, n), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    lagpu.matrix_mul_device(ctx_fast, ta.data_ptr(), k, tb.data_ptr(), n, tc.data_ptr(), n, m, k, n)
    ctx_fast.synchronize()
    c, want = tc.cpu().numpy(), _exact(a, b)
    got = np.array([[int(v) for v in row] for row in np.ldexp(c, 100)], dtype=object) * 2 ** 20
    err = np.ldexp((np.abs(got - want)).astype(np.float64), -120)
    w = np.ldexp(want.astype(np.float64), -120)
    bound = np.spacing(np.abs(w)) / 2 + 9.1 * k * 2.0 ** -64 * _scale(a, 1)[:, None] * _scale(b, 0)
    fits = np.abs(a) @ np.abs(b) >= 1.1 * 2.0 ** -8.9 * np.sqrt(k) * _scale(a, 1)[:, None] * _scale(b, 0)
    assert fits.all()  # every element is above the guard's limit
    assert np.all(err <= 1.001 * bound + 2.0 ** -99)
    if k >= 64:  # and the chain of K FMAs, the other way, is not that exact
        chain = np.zeros((m, n))
        for i in range(k):  # a product and a sum, each rounded: no worse than an FMA by more than half
            chain = chain + a[:, i:i + 1] * b[i]
        other = np.ldexp(np.abs(np.array([[int(v) for v in row] for row in np.ldexp(chain, 100)], dtype=object)
                                * 2 ** 20 - want).astype(np.float64), -120)
        assert np.sqrt((err ** 2).mean()) <= np.sqrt((other ** 2).mean()) / 2
