"""The FP64 cluster panel (panel_cluster64.cu) against the cooperative one (lu_panel.cu): the same
operations on every element, so the same bits, at the edges of its cluster sizes (128 rows per CTA,
1 to 16 CTAs), of its block sizes (128, 256 and 512 threads) and of its range (8192 rows)."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1), (3, 2), (24, 24), (31, 33), (128, 32), (129, 33), (256, 31), (257, 64), (513, 70),
          (1025, 65), (2048, 40), (2049, 40), (4096, 33), (4097, 33), (8192, 34), (8193, 40),
          (100, 300), (300, 100)]


def _factor(lagpu, ctx, a):
    lu = lagpu.LUDecomposition.new(a, ctx)
    out = lu.get_packed().data, lu.get_piv(), lu.pospivsign()
    lu.free()
    return out


@pytest.mark.parametrize("mn", SHAPES)
def test_same_bits_as_the_cooperative_panel(lagpu, ctx_fast, mn):
    a = np.random.default_rng(mn[0] * 3 + mn[1]).standard_normal(mn)
    got = _factor(lagpu, ctx_fast, a)
    ctx_fast.set_option(lagpu.OPT_CLUSTER_PANEL, 0)
    want = _factor(lagpu, ctx_fast, a)
    ctx_fast.set_option(lagpu.OPT_CLUSTER_PANEL, 1)
    assert np.array_equal(got[1], want[1]) and got[2] == want[2]
    assert np.array_equal(got[0], want[0])


@pytest.mark.parametrize("kind", ["nan", "nan_diag", "inf", "zeros", "ties", "zero_column"])
def test_pivot_rules(lagpu, ctx_fast, kind):
    n = 150
    rng = np.random.default_rng(5)
    a = rng.standard_normal((n, n))
    if kind == "nan":
        a[70, 3] = np.nan
    elif kind == "nan_diag":
        a[4, 4] = np.nan
    elif kind == "inf":
        a[100, 2] = np.inf
    elif kind == "zeros":
        a[rng.random((n, n)) < 0.7] = 0.0
    elif kind == "ties":
        a = rng.integers(-1, 2, (n, n)).astype(float)
    else:
        a[:, 40] = 0.0
    with np.errstate(all="ignore"):
        got = _factor(lagpu, ctx_fast, a)
        ctx_fast.set_option(lagpu.OPT_CLUSTER_PANEL, 0)
        want = _factor(lagpu, ctx_fast, a)
        ctx_fast.set_option(lagpu.OPT_CLUSTER_PANEL, 1)
    assert np.array_equal(got[1], want[1])
    assert np.array_equal(got[0], want[0], equal_nan=True)
    if kind in ("zeros", "zero_column"):
        assert np.array_equal(got[1], oracle.lu_factor(a).piv)


@pytest.mark.parametrize("mn", SHAPES)
def test_exact_same_bits_as_the_cooperative_panel(lagpu, ctx_exact, mn):
    """EXACT: panels in halves on the cluster (up to 4096 rows) against the whole cooperative one, and
    against the oracle where that is quick."""
    a = np.random.default_rng(mn[0] * 5 + mn[1]).standard_normal(mn)
    got = _factor(lagpu, ctx_exact, a)
    ctx_exact.set_option(lagpu.OPT_CLUSTER_PANEL, 0)
    want = _factor(lagpu, ctx_exact, a)
    ctx_exact.set_option(lagpu.OPT_CLUSTER_PANEL, 1)
    assert np.array_equal(got[1], want[1]) and got[2] == want[2]
    assert np.array_equal(got[0], want[0])
    if mn[0] * mn[1] <= 40000:
        f = oracle.lu_factor(a)
        assert np.array_equal(got[0], f.lu) and np.array_equal(got[1], f.piv)


@pytest.mark.parametrize("kind", ["nan", "nan_diag", "inf", "zeros", "ties", "zero_column", "negzero"])
def test_exact_pivot_rules(lagpu, ctx_exact, kind):
    n = 150
    rng = np.random.default_rng(6)
    a = rng.standard_normal((n, n))
    if kind == "nan":
        a[70, 3] = np.nan
    elif kind == "nan_diag":
        a[4, 4] = np.nan
    elif kind == "inf":
        a[100, 2] = np.inf
    elif kind == "zeros":
        a[rng.random((n, n)) < 0.7] = 0.0
    elif kind == "ties":
        a = rng.integers(-1, 2, (n, n)).astype(float)
    elif kind == "negzero":
        a[rng.random((n, n)) < 0.5] = -0.0
    else:
        a[:, 40] = 0.0
    with np.errstate(all="ignore"):
        got = _factor(lagpu, ctx_exact, a)
        ctx_exact.set_option(lagpu.OPT_CLUSTER_PANEL, 0)
        want = _factor(lagpu, ctx_exact, a)
        ctx_exact.set_option(lagpu.OPT_CLUSTER_PANEL, 1)
    assert np.array_equal(got[1], want[1])
    assert np.array_equal(got[0], want[0], equal_nan=True)
    assert np.array_equal(np.signbit(got[0]), np.signbit(want[0])) or np.isnan(got[0]).any()
