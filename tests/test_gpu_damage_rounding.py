"""Damage of material at rest relative to itself: the phase-field update of an undamaged, unstrained
block is exactly zero, and in FP32 too it must stay below a half unit in the last place of c = 1."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mixed", [False, True], ids=["fp32", "mixed"])
@pytest.mark.parametrize("batched", [False, True], ids=["plain", "batched"])
def test_unstrained_block_keeps_its_damage(pkg, ctx, mixed, batched):
    G = pkg.gmpm
    sp = pkg.scenes.blob(precision=G.PRECISION_FP32_FP64SVD if mixed else G.PRECISION_FP32, spin=0.0)
    scene = sp.build(ctx)
    if batched:
        batch = G.Batch(ctx, [scene], autotune=False)
        batch.substep(10)
        batch.close()
    else:
        scene.substep(10)
    assert scene.sync() == G.OK
    c = scene.read("damage")
    assert np.all(c == 1.0), (int(np.sum(c != 1.0)), float(c.min()))
