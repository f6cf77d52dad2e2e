"""Selector features at the sizes where the rows' slots of 32 columns change (4, 8, 12 and 16 of them),
in a batch whose order by size differs from the caller's."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SIZES = [257, 1, 512, 31, 128, 129, 256, 33, 384, 385, 511, 2, 32, 127, 255, 383, 16]


def test_norm_features_at_slot_edges(lagpu, ctx_fast):
    """FP32 sums of at most 512 rounded entries: relative error below 512 * 2^-24 + 2^-24, 3.1e-5, in
    log10 1.4e-5; the sum of squares of up to 512^2 entries is summed per row and then in FP64."""
    ns = np.array(SIZES)
    systems, na, nb = lagpu.batch_systems(ns, np.ones(len(ns), dtype=int))
    a = np.random.default_rng(8).standard_normal(na)
    da = torch.from_numpy(a).cuda()
    f = torch.zeros((len(ns), 16), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    lagpu.batch_features_device(ctx_fast, da.data_ptr(), systems, f.data_ptr())
    f = f.cpu().numpy()
    for i, (n, s) in enumerate(zip(ns, systems)):
        m = np.abs(a[s.a_offset:s.a_offset + n * n].reshape(n, n))
        want = np.log10([m.sum(axis=1).max(), m.sum(axis=0).max(), np.sqrt((m * m).sum()), m.max()])
        assert np.abs(f[i, 2:6] - want).max() <= 2e-5 + 1e-7 * np.abs(want).max(), n
        assert abs(f[i, 0] - np.log2(n) / 9) <= 1e-6 and f[i, 1] == 0.25
        assert np.all(np.isfinite(f[i, :12]))
