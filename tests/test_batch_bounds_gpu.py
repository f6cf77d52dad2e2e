"""Batched solves system by system: plain FP64 within the bound of its own factors, mixed within the tolerance
asked for, at sizes from 1 to 512."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
U = 2.0 ** -53
SIZES = [1, 2, 3, 16, 17, 33, 52, 65, 100, 129, 200, 257, 300, 400, 512]


def _run(lagpu, ctx, mats, rhs, mode, tol):
    systems, na, nb = lagpu.batch_systems(np.array([len(m) for m in mats]), np.array([b.shape[1] for b in rhs]))
    a, b = np.zeros(na), np.zeros(nb)
    for s, m, y in zip(systems, mats, rhs):
        a[s.a_offset:s.a_offset + m.size] = m.ravel()
        b[s.b_offset:s.b_offset + y.size] = y.ravel()
    da, db = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    dx = torch.zeros_like(db)
    torch.cuda.synchronize()
    plan = lagpu.BatchPlan(ctx, da.data_ptr(), db.data_ptr(), dx.data_ptr(), systems, mode,
                           ctas_per_sm=1, warps_per_system=8, tol=tol)
    plan.run()
    ctx.synchronize()
    x, stats = dx.cpu().numpy(), plan.stats()
    plan.free()
    return [x[s.b_offset:s.b_offset + y.size].reshape(y.shape) for s, y in zip(systems, rhs)], stats


def _systems(seed):
    rng = np.random.default_rng(seed)
    mats = [rng.standard_normal((n, n)) + 3 * np.sqrt(n) * np.eye(n)[rng.permutation(n)] for n in SIZES]
    return mats, [rng.standard_normal((n, 1 + i % 4)) for i, n in enumerate(SIZES)]


def test_fp64(lagpu, ctx_fast):
    """|A x - b| <= 4 n u |P'L| |U| |x| element by element (Higham, Accuracy and Stability of Numerical
    Algorithms, theorem 9.4, and n u for the product here), L and U those of LAPACK."""
    linalg = pytest.importorskip("scipy.linalg")
    mats, rhs = _systems(1)
    for a, x, b in zip(mats, _run(lagpu, ctx_fast, mats, rhs, lagpu.BATCH_FP64, 0.0)[0], rhs):
        p, l, u = linalg.lu(a)
        bound = (p @ np.abs(l)) @ (np.abs(u) @ np.abs(x))
        assert np.all(np.abs(a @ x - b) <= 4 * max(len(a), 2) * U * (bound + np.abs(b))), a.shape


@pytest.mark.parametrize("tol", [5e-15, 1e-12, 1e-10])
def test_mixed_meets_its_tolerance(lagpu, ctx_fast, tol):
    """The kernel's own measure within tol, and the residual formed anew within tol and the rounding errors
    of its n terms there and here (four standard deviations of u each)."""
    mats, rhs = _systems(2)
    xs, (its, eta, fallback) = _run(lagpu, ctx_fast, mats, rhs, lagpu.BATCH_MIXED, tol)
    assert np.all(eta <= tol) and np.all(fallback == 0)
    for a, x, b in zip(mats, xs, rhs):
        r = np.abs(b - a @ x).max(axis=0)
        e = (r / (np.abs(a).sum(axis=1).max() * np.abs(x).max(axis=0) + np.abs(b).max(axis=0))).max()
        assert e <= tol + 8 * np.sqrt(len(a)) * U, a.shape
