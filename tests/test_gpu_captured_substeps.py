"""A user's own CUDA graph of plain substeps, replayed after batched substeps of the same scene."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_captured_substeps_after_a_batch(pkg, ctx):
    torch = pytest.importorskip("torch")
    G = pkg.gmpm
    # two cells per substep, so that the pages of one substep are not those of the next
    sp = pkg.scenes.blob(n_side=8, velocity=(300.0, 0.0, 0.0), spin=0.0)
    scene, alone = sp.build(ctx), sp.build(ctx)
    stream = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        scene.substep(1, stream.cuda_stream)  # from the first particle buffer to the second
    batch = G.Batch(ctx, [scene], autotune=False)
    graph.replay()
    torch.cuda.synchronize()
    batch.substep(1)  # and back
    torch.cuda.synchronize()
    graph.replay()
    torch.cuda.synchronize()
    alone.substep(3)
    assert scene.sync() == G.OK and alone.sync() == G.OK
    a, b = scene.diagnostics(), alone.diagnostics()
    assert a["substeps"] == b["substeps"] == 3
    assert (a["n_blocks"], a["n_grid_blocks"]) == (b["n_blocks"], b["n_grid_blocks"])
    for array in ("block_keys", "grid_keys", "keys", "perm"):
        assert np.array_equal(scene.binning(array), alone.binning(array)), array
    batch.close()
