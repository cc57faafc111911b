"""FP64 integer products at zeros and non-finite factors: on the host with the headers the kernels use,
and cells of zero density in the kernels (GPU), which the finite check has to report."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_zero_times_nonfinite_and_zero_density(tmp_path):
    exe = tmp_path / "mul64_nonfinite_test"
    pkgdir = next(ROOT.glob("simulation-de-fluide-*_gb300"))
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I", str(pkgdir / "csrc"),
                    str(ROOT / "tests" / "cpp" / "mul64_nonfinite_test.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.gpu
@pytest.mark.parametrize("nx", [512, 130])
@pytest.mark.parametrize("force", [(0.0, 0.0), (1e-5, 0.0), (1e-5, -3e-6)])
def test_a_cell_of_zero_density_is_reported(gpu_lib, nx, force):
    ny = 40
    mask = gpu_lib.make_channel(nx, ny)
    s0 = np.zeros((ny, nx, 9))
    s0[20, 50, 0] = -1.0
    got = []
    with np.errstate(all="ignore"):
        for variant in (-1, 0):
            with gpu_lib.Solver(nx, ny, 0.7, *force, mask, precision="fp64") as s:
                s.set_variant(variant)
                s.set_populations(s0.reshape(-1))
                s.run(3)
                assert not s.check_finite()
                got.append(s.populations())
    a, b = got
    assert np.array_equal(np.isfinite(a), np.isfinite(b))
    assert np.array_equal(a[np.isfinite(a)], b[np.isfinite(b)])
