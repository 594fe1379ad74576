"""Scenes of more particles per cell than the kernels' buffers are sized for (8)."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from test_gpu_bin_paths import _expected

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("per_cell,side", [(13, 10), (27, 16), (27, 41), (64, 24)])
def test_canonical_order_of_dense_pages(pkg, per_cell, side):
    """Pages above a warp's buffer, fewer and more of them than CTAs, in shuffled order."""
    torch = pytest.importorskip("torch")
    G = pkg.gmpm
    rng = np.random.default_rng(per_cell)
    res = 64
    cells = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)
    pos = (9.5 + np.repeat(cells, per_cell, axis=0) + rng.random((per_cell * side ** 3, 3))) / res
    pos = pos[rng.permutation(len(pos))][: 1 << 20].astype(np.float32)
    n = len(pos)
    d_pos = torch.tensor(pos, device="cuda")
    perm = torch.empty(n, dtype=torch.int32, device="cuda")
    keys = torch.empty(n, dtype=torch.int32, device="cuda")
    assert G.lib().gmpm_bin_positions_noalloc(C.c_void_p(d_pos.data_ptr()), n, 1.0 / res, res, res, res,
                                              C.c_void_p(perm.data_ptr()), C.c_void_p(keys.data_ptr()), None, None) == G.OK
    torch.cuda.synchronize()
    want_perm, want_keys = _expected(pos, res)
    assert np.array_equal(keys.cpu().numpy().view(np.uint32), want_keys)
    assert np.array_equal(perm.cpu().numpy(), want_perm)
