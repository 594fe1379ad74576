"""Which scenes of a batch share launches: those that run the same kernels."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_scenes_of_both_reproducibility_settings_share_launches(pkg, ctx):
    """`deterministic` asks for nothing that P2G does not do anyway, so it does not split a batch."""
    G, S = pkg.gmpm, pkg.scenes
    specs = S.notched_bar_batch(4, seed=21, lo=6_000, hi=20_000, substeps=4)
    for k, sp in enumerate(specs):
        sp.desc.deterministic = k & 1
    scenes, alone = [sp.build(ctx) for sp in specs], [sp.build(ctx) for sp in specs]
    batch = G.Batch(ctx, scenes, autotune=False)
    batch.substep(4)
    info = batch.info()
    assert info["table_scenes"] == 4 and info["kernel_nodes"] == 23
    for a, b in zip(scenes, alone):
        b.substep(4)
        assert a.sync() == G.OK and b.sync() == G.OK
        for f in ("position", "velocity", "F", "damage"):
            assert np.array_equal(a.read(f), b.read(f)), f
    batch.close()
