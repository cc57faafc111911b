"""Several small solvers at once: the cut of a narrow grid leaves SMs to others (host), and eight
solvers that run at the same time give the numbers of one (GPU)."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_narrow_grids_take_half_the_sms(tmp_path):
    exe = tmp_path / "resident_share_test"
    pkgdir = next(ROOT.glob("simulation-de-fluide-*_gb300"))
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", str(pkgdir / "csrc"),
                    str(ROOT / "tests" / "cpp" / "resident_share_test.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny", [(5, 2), (53, 31), (127, 1), (128, 66), (97, 126), (128, 127)])
@pytest.mark.parametrize("prec", ["fp32", "fp16"])
def test_eight_solvers_at_once(gpu_lib, nx, ny, prec):
    mask = gpu_lib.make_channel(nx, ny) if ny > 8 else np.zeros(nx * ny, np.uint8)
    solvers = [gpu_lib.Solver(nx, ny, 0.6, 1e-6, 2e-7 * (k % 2), mask, precision=prec) for k in range(8)]
    want = [gpu_lib.Solver(nx, ny, 0.6, 1e-6, 2e-7 * k, mask, precision=prec) for k in range(2)]
    try:
        for s in solvers + want:
            s.init_equilibrium(1.0, 0.03, 0.01)
        for _ in range(12):
            for s in solvers:
                s.step(9)
        for s in want:
            s.set_launch(128)
            s.run(108)
        ref = [s.populations() for s in want]
        for k, s in enumerate(solvers):
            s.synchronize()
            assert np.array_equal(s.populations(), ref[k % 2])
    finally:
        for s in solvers + want:
            s.close()
