"""Host matrices whose rows are not a multiple of the device pitch are staged through a buffer of about
128 MB, several pieces for a larger matrix."""
import json
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))


@pytest.mark.parametrize("m,n", [(1001, 1002), (4094, 4099), (4097, 4099), (5803, 5802), (8195, 4097), (3, 5900001)])
def test_round_trip_in_pieces(lagpu, ctx_fast, m, n):
    """A unit triangle and entries above it factor into themselves, bit by bit. The first two shapes are
    one piece, the last has rows of a third of one."""
    a = np.random.default_rng(m).standard_normal((m, n))
    a[:, :m] = np.triu(a[:, :m], 1) + np.eye(m, min(m, n)) if m <= n else 0
    if m > n:
        a[:n] = np.triu(np.random.default_rng(n).standard_normal((n, n)), 1) + np.eye(n)
    lu = lagpu.LUDecomposition.new(a, ctx_fast)
    assert np.array_equal(lu.get_packed().data, a)
    lu.free()


CHILD = r"""
import json, sys
import numpy as np, torch
sys.path.insert(0, sys.argv[1])
import la_gpu
ctx = la_gpu.Context()
small = np.eye(130) + 1e-3
la_gpu.LUDecomposition.new(small, ctx).free()
n = 9001
a = np.eye(n)
torch.cuda.synchronize()
free = torch.cuda.mem_get_info()[0]
lu = la_gpu.LUDecomposition.new(a, ctx)
print(json.dumps(free - torch.cuda.mem_get_info()[0]))
"""


def test_device_memory_of_a_factorization(lagpu):
    """The matrix (648 MB), the digits of one update (2 x 9001 x (16 x 256 + 16) bytes, 74 MB), 128 MB
    of staging, and what the pool rounds up: 280 MB in all beyond the matrix, less than a second one."""
    r = subprocess.run([sys.executable, "-c", CHILD, os.path.join(ROOT, "rust-la_gb300")],
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    used = json.loads(r.stdout.strip().splitlines()[-1])
    assert used <= 9001 * 9004 * 8 + 280e6
