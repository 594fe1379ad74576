"""A wait of the binning's one-pass scans that runs out (tests/cpp/scan_give_up.cu): reported,
nothing written out of range, and the next binning is right."""
from __future__ import annotations

import importlib.util
import subprocess

import pytest

from conftest import PKG_DIR, ROOT

pytestmark = pytest.mark.gpu


def test_scan_that_gives_up_leaves_the_binning_usable(pkg, tmp_path):
    spec = importlib.util.spec_from_file_location("gmpm_build", PKG_DIR / "build.py")
    b = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(b)
    exe = tmp_path / "scan_give_up"
    subprocess.run([b.nvcc_path(), *b.ARCH, "-std=c++17", "-I", str(ROOT / "include"), "-I", str(b.CSRC),
                    str(ROOT / "tests" / "cpp" / "scan_give_up.cu"), str(b.LIB), "-Xlinker", f"-rpath={b.LIB.parent}",
                    "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout + r.stderr
