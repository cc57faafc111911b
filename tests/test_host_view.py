"""Which host buffers kernels may use in place (csrc/host_access.h), decided on the host: the header
the library uses, compiled against a stand-in for the CUDA runtime's pointer queries."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    cuda = Path(shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc").resolve().parents[1] / "include"
    if shutil.which("g++") is None or not (cuda / "cuda_runtime.h").exists():
        pytest.skip("no host compiler or CUDA headers")
    out = tmp_path_factory.mktemp("host_view") / "host_view_test"
    pkgdir = next(ROOT.glob("simulation-de-fluide-*_gb300"))
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", str(pkgdir / "csrc"), "-I", str(cuda),
                    str(ROOT / "tests" / "cpp" / "host_view_test.cpp"), "-o", str(out)], check=True)
    return out


@pytest.mark.parametrize("part", ["pinned", "protection", "allocation"])
def test_host_view(exe, part):
    r = subprocess.run([str(exe), part], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
