"""P2G's staging and work split at its edges, against the FP64 oracle: pages at
and around a chunk of 576 particles (one lane sums a cell, so a crowded page is
also a page of long and uneven cells), and particles given in random order, whose
previous slots lie outside the staged window of every page."""
from __future__ import annotations

import numpy as np
import pytest

from parity import errors, format_errors

pytestmark = pytest.mark.gpu

# rounding-level horizon: the tolerances of the work-split and short-horizon parity tests
TOL = {"fp64": dict(velocity=1e-9, F=1e-9, damage=1e-9, B=1e-8, volume=1e-9),
       "fp32": dict(velocity=1e-3, F=1e-4, damage=1e-4, B=2e-2, volume=1e-4)}


def _positions(name, rng, dx):
    if name == "shuffled":
        side = np.arange(20, 38) + 0.5
        lat = np.stack(np.meshgrid(side, side, side, indexing="ij"), -1).reshape(-1, 3)
        return rng.permutation(lat + rng.uniform(-0.45, 0.45, lat.shape)) * dx
    # one page (base nodes 28..31 on every axis) with its particles drawn towards one corner, and a neighbour
    crowd = 28.5 + 4.0 * rng.uniform(0.0, 1.0, (int(name), 3)) ** 1.5
    return np.concatenate([crowd, 24.5 + rng.uniform(0.0, 4.0, (37, 3))]) * dx


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("name", ["1", "575", "576", "577", "1153", "shuffled"])
def test_chunk_edges_match_oracle(pkg, ctx, oracle, name, precision):
    G, S = pkg.gmpm, pkg.scenes
    rng = np.random.default_rng(5)
    dx, res = 1.0 / 64, 64
    pos = _positions(name, rng, dx).astype(np.float32).astype(np.float64)
    vel = rng.uniform(-0.1, 0.1, pos.shape)
    d = G.reference_defaults(dx, (res, res, res))
    d.dt = 1e-4
    d.gravity[0] = d.gravity[1] = d.gravity[2] = 0.0
    d.wall_bc = 0
    d.particle_volume = dx ** 3 / 8
    S.config_material(d.materials[0], dx)
    d.precision = G.PRECISION_FP64 if precision == "fp64" else G.PRECISION_FP32
    mass = np.full(len(pos), 1000.0 * d.particle_volume)
    gpu = G.Scene(ctx, d, pos, mass, vel)
    orc = oracle.OracleScene(d, pos, mass, vel, np.zeros(len(pos), dtype=np.int32))
    gpu.substep(3)
    orc.substep(3)
    assert gpu.sync() == G.OK
    e = errors(G, gpu, orc, pos, fields=tuple(TOL[precision]))
    print(f"\n[{name} {precision} n={len(pos)}] {format_errors(e)}")
    for k, tol in TOL[precision].items():
        assert e[k] <= tol, (name, precision, k, e[k])
