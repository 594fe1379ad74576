"""One constitutive update of given particle states (deformation, damage, plastic strain, history),
against the FP64 oracle's update of the same state, particle by particle.  The states go in through a
checkpoint whose velocities, APIC matrices and stresses are zero, so the substep leaves F as given and
only the update acts on it."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HEADER = 56  # of a checkpoint file, before the scene description


def _load_state(pkg, ctx, path, precision, F, c=None, alpha=None, psi=None, yield_stress=1e9):
    """A scene of len(F) particles at rest in the given state; F as (n, 9), column-major."""
    G, S = pkg.gmpm, pkg.scenes
    n, dx, res = len(F), 1.0 / 64, 64
    pos = (20.0 + 24.0 * np.random.default_rng(2).random((n, 3))) * dx
    d = G.reference_defaults(dx, (res, res, res))
    d.dt, d.wall_bc, d.precision = 1e-6, 0, precision
    d.gravity[0] = d.gravity[1] = d.gravity[2] = 0.0
    d.particle_volume = dx ** 3 / 8
    S.config_material(d.materials[0], dx)
    d.materials[0].yield_stress = yield_stress
    scene = G.Scene(ctx, d, pos, np.full(n, 1000.0 * d.particle_volume))
    scene.save(path)
    scene.close()
    raw = bytearray(path.read_bytes())
    real = np.float64 if precision == G.PRECISION_FP64 else np.float32
    item = np.dtype(real).itemsize
    at = HEADER + C.sizeof(G.SceneDesc) + 3 * n * item  # planes: x (3), F and the plastic state (3 x 4), c, ...
    words = np.zeros((3, n, 4), dtype=real)
    f = np.asarray(F, dtype=real)
    words[0], words[1], words[2, :, 0] = f[:, :4], f[:, 4:8], f[:, 8]
    words[2, :, 1] = 0.0 if alpha is None else alpha
    words[2, :, 2] = 0.0 if psi is None else psi
    raw[at:at + words.nbytes] = words.tobytes()
    at += words.nbytes
    damage = np.ascontiguousarray(np.ones(n) if c is None else c, dtype=real)
    raw[at:at + damage.nbytes] = damage.tobytes()
    at += 2 * n * item + 4 * n + 12 * n * item  # ... m, id, v (3), B (9), stress (6)
    raw[at:at + 6 * n * item] = bytes(6 * n * item)
    path.write_bytes(raw)
    return G.Scene.load(ctx, path), d, words.astype(np.float64), damage.astype(np.float64)


def _rotations(rng, n, angle):
    axis = rng.normal(size=(n, 3))
    axis /= np.linalg.norm(axis, axis=1)[:, None]
    K = np.zeros((n, 3, 3))
    K[:, 0, 1], K[:, 0, 2], K[:, 1, 2] = -axis[:, 2], axis[:, 1], -axis[:, 0]
    K -= np.transpose(K, (0, 2, 1))
    s, c = np.sin(angle)[:, None, None], np.cos(angle)[:, None, None]
    return np.eye(3) + s * K + (1 - c) * (K @ K)


def _states(rng, n, trace_sign):
    """Deformations R exp(eps): strains on both sides of the bound |F F^T - I| = 0.1, a third of them
    unrotated, a third turned by little, a third by any angle."""
    eps = rng.normal(size=(n, 3, 3))
    eps += np.transpose(eps, (0, 2, 1))
    eps -= np.trace(eps, axis1=1, axis2=2)[:, None, None] / 3 * np.eye(3)
    eps *= (rng.uniform(0.003, 0.06, n) / np.linalg.norm(eps, axis=(1, 2)))[:, None, None]
    eps += (trace_sign * rng.uniform(0.004, 0.06, n) / 3)[:, None, None] * np.eye(3)
    w, V = np.linalg.eigh(eps)
    U = (V * np.exp(w)[:, None, :]) @ np.transpose(V, (0, 2, 1))
    angle = np.where(np.arange(n) % 3 == 0, 0.0, np.where(np.arange(n) % 3 == 1, rng.uniform(0, 0.05, n),
                                                          rng.uniform(0, np.pi, n)))
    return np.transpose(U @ _rotations(rng, n, angle), (0, 2, 1)).reshape(n, 9)  # column-major


@pytest.mark.parametrize("precision", [0, 1, 2], ids=["fp32", "mixed", "fp64"])
def test_reflected_deformation_is_reported(pkg, ctx, tmp_path, precision):
    """det F < 0 with singular values near 1 (a step far above stability): the stress is not a number
    and the next substep says so, as for any other state without a stress."""
    G = pkg.gmpm
    prec = (G.PRECISION_FP32, G.PRECISION_FP32_FP64SVD, G.PRECISION_FP64)[precision]
    rng = np.random.default_rng(3)
    F = _states(rng, 1200, -1.0) * np.where(np.arange(9) >= 6, -1.0, 1.0)
    M = F.reshape(-1, 3, 3)  # transposed
    F = F[np.linalg.norm(np.transpose(M, (0, 2, 1)) @ M - np.eye(3), axis=(1, 2)) < 0.09]
    scene, *_ = _load_state(pkg, ctx, tmp_path / "state.gmpm", prec, F)
    scene.substep(2)
    scene.sync()
    assert scene.diagnostics()["flags"] & G.FLAG_NONFINITE


# A strain is known to the rounding of F F^T: entries of F F^T - I sum five products of FP32 numbers up to 2 (a large
# rotation), 5 * 4 * 2^-24 = 1.2e-6, half of it in the strain.
STRAIN = 1e-6


@pytest.mark.parametrize("trace", [1.0, -1.0], ids=["expanded", "compressed"])
@pytest.mark.parametrize("yields", [False, True], ids=["elastic", "yielding"])
@pytest.mark.parametrize("mixed", [False, True], ids=["fp32", "mixed"])
def test_update_matches_oracle(pkg, ctx, oracle, tmp_path, mixed, yields, trace):
    G = pkg.gmpm
    rng = np.random.default_rng(7)
    n = 3000
    scene, d, words, c_old = _load_state(
        pkg, ctx, tmp_path / "state.gmpm", G.PRECISION_FP32_FP64SVD if mixed else G.PRECISION_FP32,
        _states(rng, n, trace), c=rng.uniform(0.3, 1.0, n), alpha=rng.uniform(0.0, 0.02, n),
        psi=rng.uniform(0.0, 30.0, n), yield_stress=200.0 if yields else 1e9)
    scene.substep(1)
    assert scene.sync() == G.OK
    got = {f: scene.read(f) for f in ("F", "alpha", "psi_max", "FP", "stress", "volume", "damage")}
    m, V0 = d.materials[0], d.particle_volume
    g = c_old ** 2 * (1 - m.theta) + m.theta
    io = np.concatenate([words[0], words[1], words[2, :, :1], g[:, None], words[2, :, 1:2],
                         got["damage"][:, None], words[2, :, 2:3]], axis=1)
    want = np.empty((n, 23))
    lib, dp = oracle.lib(), C.POINTER(C.c_double)
    for p in range(n):
        lib.orc_constitutive(C.byref(m), V0, d.dx, io[p].ctypes.data_as(dp), want[p].ctypes.data_as(dp))
    # the strain's error: its rounding, and through the return map, which scales the deviator's direction by the
    # yield excess, the excess over the deviator's size times that
    E, nu = m.youngs_modulus, m.poisson_ratio
    lam, mu = E * nu / ((1 + nu) * (1 - 2 * nu)), E / (2 * (1 + nu))
    K = lam + 2 * mu
    eps = np.log(np.linalg.svd(io[:, :9].reshape(n, 3, 3), compute_uv=False))
    tr = eps.sum(axis=1)
    tt = lam * tr[:, None] + 2 * mu * eps
    tn = g * 2 * mu * np.linalg.norm(eps - tr[:, None] / 3, axis=1)
    tsum = tt.sum(axis=1)
    err = np.full(n, STRAIN)
    d_alpha = np.zeros(n)
    if yields:
        moved = ~np.all(want[:, :9] == io[:, :9], axis=1)
        assert moved.all()
        y = np.linalg.norm(tt, axis=1)
        err *= 4 + 2 * y / tn
        dl = np.abs(want[:, 10] - io[:, 10])
        d_alpha = 2 * dl * STRAIN * (3 * K / np.abs(tsum) + 2 * K / (y - np.sqrt(2 / 3) * g * (200.0 + 0.1 * E * io[:, 10])))
    d_psi = 0.6 * K * err + 1e-5 * want[:, 11]
    rate = (want[:, 12] - 1) / np.maximum(want[:, 11], 1e-9)
    checks = {"F": (np.abs(got["F"] - want[:, :9]).max(axis=1), 2 * err),
              "alpha": (np.abs(got["alpha"] - want[:, 10]), d_alpha + 1e-6),
              "psi_max": (np.abs(got["psi_max"] - want[:, 11]), d_psi),
              "FP": (np.abs(got["FP"] - want[:, 12]), rate * d_psi + (d_alpha + 1e-5) * want[:, 12]),
              "volume": (np.abs(got["volume"] - want[:, 22]), V0 * (4 * err + 1e-6))}
    s = want[:, 13:22].reshape(n, 3, 3)
    six = np.stack([s[:, 0, 0], s[:, 1, 1], s[:, 2, 2], (s[:, 0, 1] + s[:, 1, 0]) / 2, (s[:, 0, 2] + s[:, 2, 0]) / 2,
                    (s[:, 1, 2] + s[:, 2, 1]) / 2], axis=1)
    checks["stress"] = (np.abs(got["stress"] - six).max(axis=1), 4 * K * V0 * err)
    print("".join(f"\n  {k}: largest share of its bound {np.max(e / b):.3f}" for k, (e, b) in checks.items()))
    for k, (e, b) in checks.items():
        assert np.all(e <= b), (k, int(np.argmax(e / b)), float(np.max(e / b)))


def test_fallback_threshold_above_the_small_strains(pkg, ctx, tmp_path):
    """A threshold of 0.9 sends no small strain to FP64 (their singular values differ by less), so it changes
    nothing; one above 1 sends every state there."""
    G = pkg.gmpm
    F = _states(np.random.default_rng(11), 1500, 1.0)
    M = F.reshape(-1, 3, 3)
    F = F[np.linalg.norm(np.transpose(M, (0, 2, 1)) @ M - np.eye(3), axis=(1, 2)) < 0.09]
    stress = {}
    for ratio in (1e-3, 0.9, 0.999, 1.1):
        path = tmp_path / "state.gmpm"
        scene, d, *_ = _load_state(pkg, ctx, path, G.PRECISION_FP32_FP64SVD, F)
        scene.close()
        raw = bytearray(path.read_bytes())
        at = HEADER + G.SceneDesc.svd_fallback_ratio.offset
        raw[at:at + 8] = np.float64(ratio).tobytes()
        path.write_bytes(raw)
        scene = G.Scene.load(ctx, path)
        scene.substep(1)
        assert scene.sync() == G.OK
        stress[ratio] = scene.read("stress")
    assert np.array_equal(stress[0.9], stress[1e-3])
    assert not np.array_equal(stress[1.1], stress[1e-3])
    assert np.array_equal(stress[0.999], stress[1.1])  # strains of 0.003 and more are below it
