"""The batched solver's panel (rows in registers, one to eight warps) and its triangular solves (a warp
for the chain, one for the tiles, the others for the rows) at the sizes where their splits change:
blocks of 16, tiles read directly below n = 52, one and two rows per thread, more rows than registers
hold; and values far outside the range in which a quotient is taken without a division."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 15, 16, 17, 31, 33, 47, 51, 52, 53, 64, 65, 81, 127, 128, 129, 200, 256, 257, 300, 511, 512]


def _run(lagpu, ctx, mats, rhs, mode, warps):
    ns = np.array([m.shape[0] for m in mats])
    rs = np.array([b.shape[1] for b in rhs])
    systems, na, nb = lagpu.batch_systems(ns, rs)
    a, b = np.zeros(na), np.zeros(nb)
    for s, m, y in zip(systems, mats, rhs):
        a[s.a_offset:s.a_offset + m.size] = m.ravel()
        b[s.b_offset:s.b_offset + y.size] = y.ravel()
    da, db = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    dx = torch.zeros_like(db)
    torch.cuda.synchronize()
    plan = lagpu.BatchPlan(ctx, da.data_ptr(), db.data_ptr(), dx.data_ptr(), systems, mode,
                           ctas_per_sm=1, warps_per_system=warps, tol=5e-15)
    plan.run()
    ctx.synchronize()
    x = dx.cpu().numpy()
    plan.free()
    return [x[s.b_offset:s.b_offset + y.size].reshape(y.shape) for s, y in zip(systems, rhs)]


def _backward(a, x, b):
    r = np.abs(b - a @ x).max(axis=0)
    return (r / (np.abs(a).sum(axis=1).max() * np.abs(x).max(axis=0) + np.abs(b).max(axis=0))).max()


def _systems(seed):
    rng = np.random.default_rng(seed)
    mats = [rng.standard_normal((n, n)) + 3 * np.sqrt(n) * np.eye(n)[rng.permutation(n)] for n in SIZES]
    return mats, [rng.standard_normal((n, 1 + i % 4)) for i, n in enumerate(SIZES)]


@pytest.mark.parametrize("warps", [2, 4, 8])
@pytest.mark.parametrize("mixed", [0, 1])
def test_sizes(lagpu, ctx_fast, warps, mixed):
    """Partial pivoting without growth: backward error below n u times a small constant, 512 * 1.1e-16 *
    4 = 2.3e-13 in the worst case, about 1e-15 as a rule; refined systems meet the asked 5e-15."""
    mats, rhs = _systems(warps + 10 * mixed)
    mode = lagpu.BATCH_MIXED if mixed else lagpu.BATCH_FP64
    for a, x, b in zip(mats, _run(lagpu, ctx_fast, mats, rhs, mode, warps), rhs):
        assert _backward(a, x, b) <= 2.3e-13, a.shape


@pytest.mark.parametrize("ea,eb", [(700, -200), (-600, 100), (520, 0), (-520, 400), (0, -700)])
def test_far_ranges(lagpu, ctx_fast, ea, eb):
    """Scaling by powers of two changes no rounding of the factorization, and of the solves only a
    quotient's last bit where it is taken by a division: 16 kappa u at kappa <= 50 is 1e-13."""
    mats, rhs = _systems(3)
    x0 = _run(lagpu, ctx_fast, mats, rhs, lagpu.BATCH_FP64, 4)
    x1 = _run(lagpu, ctx_fast, [np.ldexp(m, ea) for m in mats], [np.ldexp(b, eb) for b in rhs],
              lagpu.BATCH_FP64, 4)
    for p, q in zip(x0, x1):
        q = np.ldexp(q, ea - eb)
        assert np.abs(p - q).max() <= 1e-13 * np.abs(p).max()


def test_singular_and_sparse(lagpu, ctx_fast):
    """Zero pivots give infinities or NaN as a division does, unit columns keep exact zeros."""
    n = 70
    rng = np.random.default_rng(4)
    a = np.triu(rng.standard_normal((n, n))) + 8 * np.eye(n)
    e = np.zeros((n, 3))
    e[[0, 20, 69], [0, 1, 2]] = 1.0
    s = a.copy()
    s[:, 40] = 0.0
    x, y = _run(lagpu, ctx_fast, [a, s], [e, rng.standard_normal((n, 1))], lagpu.BATCH_FP64, 4)
    assert np.all(x[1:, 0] == 0) and np.all(x[21:, 1] == 0)
    assert _backward(a, x, e) <= 1e-14
    assert not np.all(np.isfinite(y))
