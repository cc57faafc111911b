"""FP64 on the integer units: the multiplication against the host processor's, and the step kernels
that use it against those with the hardware's multiplications, bit for bit, also where the
integer ones hand over (zeros, tiny and huge values, infinities and NaNs)."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_products_equal_the_processors(tmp_path):
    exe = tmp_path / "mul64_test"
    pkgdir = next(ROOT.glob("simulation-de-fluide-*_gb300"))
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", str(pkgdir / "csrc"),
                    str(ROOT / "tests" / "cpp" / "mul64_test.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr


def state(kind, nx, ny, mask, pkg):
    s = pkg.workloads.seeded_state(3, 1e-2, nx, ny, mask, np.float64).reshape(ny, nx, 9)
    if kind == "zero":
        s[:] = 0.0
    elif kind == "tiny":  # products below the window, and below the normal range
        s[:] = 0.0
        s[5:9, 20:40] = 1e-150
        s[20:24, 60:90, 1] = 1e-310
    elif kind == "large":
        s[10, 50] = [0, 1e200, 0, -1e200, 0, 0, 0, 0, 0]
    elif kind == "nonfinite":
        s[10, 50, 3] = np.inf
        s[12, 90, 5] = np.nan
    return s.reshape(-1)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["seeded", "zero", "tiny", "large", "nonfinite"])
@pytest.mark.parametrize("nx,ny", [(512, 40), (300, 40), (130, 40)])
@pytest.mark.parametrize("force", [(0.0, 0.0), (1e-5, 0.0), (1e-5, -3e-6)])
def test_integer_and_hardware_kernels_agree(gpu_lib, kind, nx, ny, force):
    mask = gpu_lib.geometry.add_block(gpu_lib.make_channel(nx, ny), nx, 30, 41, 9, 17)
    s0 = state(kind, nx, ny, mask, gpu_lib)
    got = []
    with np.errstate(all="ignore"):
        for variant in (-1, 0):
            with gpu_lib.Solver(nx, ny, 0.7, *force, mask, precision="fp64") as s:
                s.set_variant(variant)
                s.set_populations(s0)
                s.run(6)
                got.append(s.populations())
        with gpu_lib.Strips(nx, ny, 0.7, *force, mask, 3, precision="fp64") as h:
            h.set_populations(s0)
            h.run(6)
            got.append(h.populations())
        spec = {"nx": nx, "ny": ny, "mask": mask, "tau": 0.7, "fx": force[0], "fy": force[1]}
        with gpu_lib.Batch([spec, spec], precision="fp64") as b:
            b.set_populations(0, s0)
            b.set_populations(1, s0)
            b.run(6)
            got += [b.populations(0), b.populations(1)]
    for g in got[:1] + got[2:]:
        assert np.array_equal(np.isfinite(g), np.isfinite(got[1]))
        assert np.array_equal(g[np.isfinite(g)], got[1][np.isfinite(g)])


@pytest.mark.gpu
def test_adjoint_forward_with_integer_products(gpu_lib):
    """alpha = 0 is the plain method, bit for bit, from a state with zeros and tiny values."""
    nx, ny = 300, 40
    mask = gpu_lib.make_channel(nx, ny)
    for kind in ("seeded", "tiny"):
        s0 = state(kind, nx, ny, mask, gpu_lib)
        with gpu_lib.Adjoint(nx, ny, 0.7, 1e-5, 0.0, mask, precision="fp64", checkpoint_every=4) as a, \
                gpu_lib.Solver(nx, ny, 0.7, 1e-5, 0.0, mask, precision="fp64") as s:
            a.forward(6, 2, s0)
            s.set_variant(0)
            s.set_populations(s0)
            s.run(6)
            assert np.array_equal(a.populations(), s.populations())
