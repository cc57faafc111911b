"""The exact collision's short forms where products underflow: against the literal collision on the
host, and runs from rest under tiny forces against the oracle (GPU), value for value."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_short_forms_equal_the_literal_collision(tmp_path):
    exe = tmp_path / "collide_tiny_test"
    pkgdir = next(ROOT.glob("simulation-de-fluide-*_gb300"))
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I", str(pkgdir / "csrc"),
                    str(ROOT / "tests" / "cpp" / "collide_tiny_test.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.gpu
@pytest.mark.parametrize("real,prec,fx", [("f32", "fp32", 1e-20), ("f32", "fp32", -3e-22), ("f64", "fp64", 1e-160)])
@pytest.mark.parametrize("variant", [-1, 0, 12])
def test_from_rest_under_a_tiny_force(gpu_lib, orc, real, prec, fx, variant):
    nx, ny, steps = 300, 33, 8
    mask = gpu_lib.make_channel(nx, ny)
    dt = np.float32 if real == "f32" else np.float64
    s0 = np.zeros(nx * ny * 9, dt)
    with gpu_lib.Solver(nx, ny, 0.7, fx, 0.0, mask, precision=prec) as s:
        s.set_variant(variant)
        s.set_populations(s0)
        s.run(steps)
        got = s.populations()
    want = orc.v0_run(nx, ny, mask, float(dt(0.7)), fx, 0.0, s0, steps, real=real)
    assert np.array_equal(got, want)
