"""A kernel launched by launch_dependent is resident while its predecessors still write its inputs, so
no pointer parameter may promise the compiler that the data is read-only for the kernel's whole life
(const with __restrict__ allows the non-coherent load path): checked on the sources.  The exception is
G2P's scene block, which no kernel writes but for the time step, read through scene_dt."""
from __future__ import annotations

import re

from conftest import PKG_DIR


def _dependent_kernels():
    for path in sorted((PKG_DIR / "csrc").glob("*.cu")):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for m in re.finditer(r"__global__[^{;]*?\b(k_\w+)\s*\(([^{;]*)\)\s*\{\s*([^;]*;)", text):
            if "depend_on_previous()" in m.group(3):
                yield path.name, m.group(1), m.group(2)


def test_dependent_kernels_promise_no_read_only_inputs():
    kernels = list(_dependent_kernels())
    launched = set()
    for path in (PKG_DIR / "csrc").glob("*.cu"):
        for call in re.findall(r"launch_dependent\(([^;]*?),\s*(?:dim3|gb|one|col|kx)\b", path.read_text()):
            launched |= set(re.findall(r"\bk_\w+", call))
    names = {name for _, name, _ in kernels}
    assert launched <= names and len(names) >= 20, (launched - names, len(names))  # each waits first
    block = re.compile(r"const SceneDev<\w+>\* __restrict__ \w+")
    assert not [(f, k) for f, k, params in kernels
                if "__restrict__" in (block.sub("", params) if k == "k_g2p" else params)]
    g2p = (PKG_DIR / "csrc" / "g2p.cu").read_text()
    body = g2p[g2p.index("void g2p_body("):g2p.index("void advance_time_body(")]
    assert "scene_dt(sc)" in body and "->dt" not in body.replace("->dt_", "")
