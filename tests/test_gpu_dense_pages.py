"""Scenes of more particles per cell than the kernels' buffers are sized for (8)."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from parity import errors, format_errors
from test_gpu_bin_paths import _expected
from test_gpu_p2g_chunks import TOL

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


def _dense(name, rng):
    """Base nodes 20.. of a 64^3 grid: whole pages start at multiples of 4."""
    if name.startswith("cell"):  # one cell above a chunk, in a page of few others
        return np.concatenate([32.5 + rng.random((int(name[4:]), 3)), 30.5 + 8.0 * rng.random((300, 3))])
    if name == "corner":  # a page's particles in its last cells only, some cells of it empty
        return np.concatenate([34.5 + 2.0 * rng.random((2000, 3)), 28.5 + 1.0 * rng.random((40, 3))])
    per_cell = int(name)
    cells = np.stack(np.meshgrid(*[np.arange(20, 29)] * 3, indexing="ij"), -1).reshape(-1, 3)
    return 0.5 + np.repeat(cells, per_cell, axis=0) + rng.random((per_cell * len(cells), 3))


@pytest.mark.parametrize("batched", [False, True], ids=["plain", "batched"])
@pytest.mark.parametrize("name", ["9", "10", "19", "37", "73", "cell577", "cell1800", "corner"])
def test_p2g_of_dense_pages_matches_oracle(pkg, ctx, oracle, name, batched):
    """Pages that are cut into runs of 32, 16, 8 and fewer cells, whose particles several lanes share."""
    G, S = pkg.gmpm, pkg.scenes
    rng = np.random.default_rng(17)
    dx, res = 1.0 / 64, 64
    pos = rng.permutation(_dense(name, rng) * dx).astype(np.float32).astype(np.float64)
    vel = rng.uniform(-0.1, 0.1, pos.shape)
    d = G.reference_defaults(dx, (res, res, res))
    d.dt = 1e-4
    d.gravity[0] = d.gravity[1] = d.gravity[2] = 0.0
    d.wall_bc = 0
    d.particle_volume = dx ** 3 / 8
    S.config_material(d.materials[0], dx)
    mass = np.full(len(pos), 1000.0 * d.particle_volume)
    gpu = G.Scene(ctx, d, pos, mass, vel)
    again = G.Scene(ctx, d, pos, mass, vel)
    orc = oracle.OracleScene(d, pos, mass, vel, np.zeros(len(pos), dtype=np.int32))
    if batched:
        batch = G.Batch(ctx, [gpu], autotune=False)
        batch.substep(3)
        batch.close()
    else:
        gpu.substep(3)
    again.substep(3)
    orc.substep(3)
    assert gpu.sync() == G.OK
    e = errors(G, gpu, orc, pos, fields=tuple(TOL["fp32"]))
    print(f"\n[{name} n={len(pos)}] {format_errors(e)}")
    for k, tol in TOL["fp32"].items():
        assert e[k] <= tol, (name, k, e[k])
    for f in ("position", "velocity", "F", "damage"):  # to the bit, with every launch shape
        assert np.array_equal(gpu.read(f), again.read(f)), f
