"""FP32 constitutive update on both sides of the small-strain bound (the polynomial path is
taken up to |F F^T - I| = 0.1, the SVD beyond), elastic and yielding, against the FP64 oracle:
a block under a uniform velocity gradient, which one substep turns into F = I + dt grad v."""
from __future__ import annotations

import numpy as np
import pytest

from parity import errors, format_errors

pytestmark = pytest.mark.gpu

# F carries rounding of 1e-7; a stress of strain s has s * E to resolve it against (s >= 1e-3 here)
TOL = dict(F=1e-5, volume=1e-5, damage=1e-4, stress=2e-3)


@pytest.mark.parametrize("yields", [False, True], ids=["elastic", "yielding"])
@pytest.mark.parametrize("strain", [0.001, 0.03, 0.049, 0.051, 0.2])
def test_strain_bound_matches_oracle(pkg, ctx, oracle, strain, yields):
    G, S = pkg.gmpm, pkg.scenes
    sp = S.blob(n_side=8, precision=G.PRECISION_FP32, velocity=(0.0, 0.0, 0.0), spin=0.0)
    d = sp.desc
    if yields:
        d.materials[0].yield_stress = 200.0
    # |grad v| dt = strain: stretch along x, half of it back along y, some shear and spin
    L = np.array([[1.0, 0.4, 0.0], [-0.2, -0.5, 0.3], [0.1, 0.0, 0.2]])
    L *= strain / (np.linalg.norm(L + L.T) / 2 * d.dt)
    vel = (sp.positions - sp.positions.mean(axis=0)) @ L.T
    gpu = G.Scene(ctx, d, sp.positions, sp.masses, vel, sp.material_ids)
    orc = oracle.OracleScene(d, sp.positions, sp.masses, vel, sp.material_ids)
    gpu.substep(1)
    orc.substep(1)
    assert gpu.sync() == G.OK
    e = errors(G, gpu, orc, sp.positions, fields=tuple(TOL))
    print(f"\n[strain {strain} yields {yields}] {format_errors(e)}")
    for k, tol in TOL.items():
        assert e[k] <= tol, (strain, yields, k, e[k])
