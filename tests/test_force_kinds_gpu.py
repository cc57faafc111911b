"""The exact collision's force kinds and the large-grid FP32 ring against the oracle (GPU): no
force, force along x alone, along y alone and along both, on every kind of step kernel, equal
value for value (the collision is bit-exact, so the tolerance is zero)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("real,prec", [("f32", "fp32"), ("f64", "fp64")])
@pytest.mark.parametrize("force", [(0.0, 0.0), (1e-5, 0.0), (0.0, 1e-5), (1e-5, 2e-6)])
@pytest.mark.parametrize("variant", [-1, 0, 7, 12, 19])
def test_force_kinds(gpu_lib, orc, real, prec, force, variant):
    nx, ny, steps = 259, 33, 12
    mask = gpu_lib.geometry.add_block(gpu_lib.make_channel(nx, ny), nx, 30, 41, 9, 17)
    dt = np.float32 if real == "f32" else np.float64
    s0 = gpu_lib.workloads.seeded_state(5, 1e-2, nx, ny, mask, dt)
    with gpu_lib.Solver(nx, ny, 0.7, *force, mask, precision=prec) as s:
        s.set_variant(variant)
        s.set_populations(s0)
        s.run(steps)
        got = s.populations()
    want = orc.v0_run(nx, ny, mask, float(dt(0.7)), *force, s0, steps, real=real)
    assert np.array_equal(got, want)


@pytest.mark.parametrize("nx,ny", [(2049, 1025), (8191, 257), (4096, 512), (8200, 5650)])
def test_large_fp32_ring_equals_direct(gpu_lib, nx, ny):
    """At least 2^21 cells: the automatic ring (256-cell tiles, ragged last tile) against the
    direct kernel."""
    mask = gpu_lib.geometry.add_block(gpu_lib.make_channel(nx, ny), nx, 250, 262, 90, 120)
    s0 = gpu_lib.workloads.seeded_state(9, 1e-3, nx, ny, mask, np.float32)
    got = []
    for variant in (-1, 0):
        with gpu_lib.Solver(nx, ny, 0.6, 1e-6, 0.0, mask) as s:
            s.set_variant(variant)
            s.set_populations(s0)
            s.run(5)
            got.append(s.populations())
    assert np.array_equal(*got)


@pytest.mark.parametrize("form", ["fp16", "bf16"])
@pytest.mark.parametrize("force", [(0.0, 0.0), (1e-5, 0.0), (0.0, 1e-5), (1e-5, 2e-6)])
@pytest.mark.parametrize("nx,ny,open_x", [(259, 33, False), (259, 33, True), (1500, 640, False)])
def test_force_kinds_16bit(gpu_lib, form, force, nx, ny, open_x):
    """16-bit storage: the rings and the resident kernel by force kind against the direct kernel,
    which evaluates every force term; equal numbers (zeros may differ in sign)."""
    mask = gpu_lib.geometry.add_block(gpu_lib.make_channel(nx, ny), nx, 30, 41, 9, 17)
    got = []
    for variant in (0, -1, 12, 17, 19, 20):
        with gpu_lib.Solver(nx, ny, 0.7, *force, mask, precision=form) as s:
            if open_x:
                s.set_inflow_outflow(0.05)
            s.set_variant(variant)
            s.init_equilibrium(1.0, 0.05, 0.01)
            s.run(9)
            got.append(s.populations())
    for g in got[1:]:
        assert np.array_equal(g, got[0])
