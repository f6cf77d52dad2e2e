"""FAST LU of more rows than one cluster's panel takes (8192): the cooperative panel takes a block of 64
columns in one piece, and the cluster panel takes over once the rows below the diagonal fit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n", [(8193, 64), (9000, 33), (20000, 64)])
def test_one_panel_and_no_updates(lagpu, ctx_fast, m, n):
    a = np.random.default_rng(m + n).standard_normal((m, n))
    before = ctx_fast.kernel_launches()
    lu = lagpu.LUDecomposition.new(a, ctx_fast)
    assert ctx_fast.kernel_launches() - before == 2  # the panel; the permutation, sign and zero flag
    lu.free()


@pytest.mark.parametrize("m,n", [(8200, 70), (8224, 130), (8320, 200)])
def test_same_bits_as_cooperative_panels_throughout(lagpu, ctx_fast, m, n):
    a = np.random.default_rng(m * 3 + n).standard_normal((m, n))
    out = []
    for cluster in (1, 0):
        ctx_fast.set_option(lagpu.OPT_CLUSTER_PANEL, cluster)
        lu = lagpu.LUDecomposition.new(a, ctx_fast)
        out.append((lu.get_packed().data, lu.get_piv(), lu.pospivsign()))
        lu.free()
    ctx_fast.set_option(lagpu.OPT_CLUSTER_PANEL, 1)
    assert np.array_equal(out[0][1], out[1][1]) and out[0][2] == out[1][2]
    assert np.array_equal(out[0][0], out[1][0])
