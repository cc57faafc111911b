"""The resident kernel's tiles and edge exchange, modelled on the host with the header the kernel
uses (csrc/resident_layout.h)."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_every_pull_is_served(tmp_path):
    exe = tmp_path / "resident_layout_test"
    pkgdir = next(ROOT.glob("simulation-de-fluide-*_gb300"))
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", str(pkgdir / "csrc"),
                    str(ROOT / "tests" / "cpp" / "resident_layout_test.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
