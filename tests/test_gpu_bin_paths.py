"""Binning's dispatch edges: two or eight particles per thread, the key pass of few and of many
positions, pages with few and with many cells out of order, scans of one and of several tiles."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _positions(n, res, shuffled, rng):
    side = min((n / 8.0) ** (1.0 / 3.0), res - 8.0)
    pos = (4.0 + side * rng.uniform(0.0, 1.0, (n, 3))) / res
    if not shuffled:  # by cell, so that few slots are out of order
        base = (pos * res + 0.5).astype(np.int64)
        pos = pos[np.lexsort((base[:, 2], base[:, 1], base[:, 0]))]
    return pos.astype(np.float32)


def _expected(pos, res):
    base = (pos.astype(np.float64) * res + 0.5).astype(np.int64) - 1
    key = np.zeros(len(pos), dtype=np.uint32)
    for bit in range(8):
        for a in range(3):
            key |= (((base[:, a] >> (2 + bit)) & 1) << (3 * bit + 2 - a)).astype(np.uint32)
    key = (key << 6) | ((base[:, 0] & 3) << 4 | (base[:, 1] & 3) << 2 | (base[:, 2] & 3)).astype(np.uint32)
    perm = np.argsort(key, kind="stable")
    return perm.astype(np.int32), key[perm]


@pytest.mark.parametrize("shuffled", [False, True], ids=["by_cell", "shuffled"])
@pytest.mark.parametrize("n,res", [(1, 8), (257, 16), (65_535, 64), (65_536, 128), (300_001, 128)])
def test_noalloc_paths(pkg, n, res, shuffled):
    torch = pytest.importorskip("torch")
    G = pkg.gmpm
    pos = _positions(n, res, shuffled, np.random.default_rng(n))
    d_pos = torch.tensor(pos, device="cuda")
    perm = torch.empty(n, dtype=torch.int32, device="cuda")
    keys = torch.empty(n, dtype=torch.int32, device="cuda")
    assert G.lib().gmpm_bin_positions_noalloc(C.c_void_p(d_pos.data_ptr()), n, 1.0 / res, res, res, res,
                                              C.c_void_p(perm.data_ptr()), C.c_void_p(keys.data_ptr()), None, None) == G.OK
    torch.cuda.synchronize()
    want_perm, want_keys = _expected(pos, res)
    assert np.array_equal(keys.cpu().numpy().view(np.uint32), want_keys)
    assert np.array_equal(perm.cpu().numpy(), want_perm)


@pytest.mark.parametrize("n,res", [(606_207, 128), (606_208, 160)])
def test_scene_paths_and_batch_handover(pkg, ctx, n, res):
    """A scene around the size where a thread takes eight particles, binned by itself, after a batched
    substep (whose binning leaves its flags set) and after a plain one."""
    G, S = pkg.gmpm, pkg.scenes
    pos = _positions(n, res, False, np.random.default_rng(n)).astype(np.float64)
    d = G.reference_defaults(1.0 / res, (res, res, res))
    d.dt, d.wall_bc = 1e-5, 0
    S.config_material(d.materials[0], 1.0 / res)
    scene = G.Scene(ctx, d, pos, np.full(n, 1e-6))
    batch = G.Batch(ctx, [scene], autotune=False)
    for step in (lambda: None, lambda: batch.substep(1), lambda: scene.substep(1)):
        step()
        assert scene.sync() == G.OK
        before = scene.read("position", order=G.ORDER_INTERNAL, dtype=G.DTYPE_F32).astype(np.float64)
        scene.rebin()
        want_perm, want_keys = _expected(before, res)
        assert np.array_equal(scene.binning("keys"), want_keys)
        assert np.array_equal(scene.binning("perm"), want_perm)
    batch.close()
