"""Open outlet beside solid cells of the column before it (GPU). An outlet cell takes the populations
that cell nx - 2 of its row receives; where that cell is solid it holds none, so a population that
would bounce back from it is zero, as in the reference's pull kernels, and never what a step kernel
happened to store in a solid slot. Against the oracle's pull steps value for value (FP32 / FP64,
every kind of step kernel, the strip engine, the moment pass), and 16-bit storage kernel against
kernel."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NY, STEPS, U = 33, 9, 0.05


def geometry(pkg, nx):
    m = pkg.make_channel(nx, NY).reshape(NY, nx).copy()
    m[1, nx - 2] = 1  # touches the wall: the corner between it, the wall and the outlet
    m[NY - 2, nx - 4:nx - 1] = 1
    m[15:18, nx - 2] = 1  # free of the outlet column
    m[10, nx - 1] = m[9, nx - 2] = 1  # diagonal pair
    m[22, nx - 1] = m[23, nx - 2] = m[21, nx - 2] = 1
    m[12:20, 8:12] = 1
    return m.reshape(-1)


def seeded(pkg, nx, mask, dt):
    return pkg.workloads.seeded_state(3, 1e-2, nx, NY, mask, dt)


@pytest.mark.parametrize("real,prec", [("f32", "fp32"), ("f64", "fp64")])
@pytest.mark.parametrize("nx", [40, 130, 259, 515])
@pytest.mark.parametrize("variant", [-1, 0, 1, 4, 7, 9, 12, 17, 19, 20])
def test_solver_equals_the_oracle(gpu_lib, orc, real, prec, nx, variant):
    dt = np.float32 if real == "f32" else np.float64
    mask, fx = geometry(gpu_lib, nx), 1e-6
    s0 = seeded(gpu_lib, nx, mask, dt)
    r = orc.s_to_r(nx, NY, mask, s0, open_x=True, real=real)
    r = orc.pull_run(nx, NY, mask, float(dt(0.7)), fx, 0.0, r, STEPS, open_x=True, u_in=U, real=real)
    want = orc.r_to_s(nx, NY, mask, r, open_x=True, u_in=U, real=real)
    with gpu_lib.Solver(nx, NY, 0.7, fx, 0.0, mask, precision=prec) as s:
        s.set_inflow_outflow(U)
        s.set_variant(variant)
        s.set_populations(s0)
        s.run(STEPS)
        assert np.array_equal(s.populations(), want)
        for a, b in zip(s.macroscopic(), orc.macroscopic(nx, NY, mask, fx, 0.0, want, real=real)):
            assert np.array_equal(a, b)
        assert np.array_equal(s.populations_at(nx - 1, 1), want.reshape(NY, nx, 9)[1, nx - 1])


@pytest.mark.parametrize("prec", ["fp32", "fp64", "fp16", "bf16"])
@pytest.mark.parametrize("nx", [130, 515])
def test_kernels_agree(gpu_lib, prec, nx):
    """Runs of many steps, of single steps and the strips: the same populations."""
    dt = np.float64 if prec == "fp64" else np.float32
    mask = geometry(gpu_lib, nx)
    s0 = seeded(gpu_lib, nx, mask, dt)
    got = []
    for how in ("run", "single", 0, 4, 9, 12, 17, 19, 20, "strips"):
        if how == "strips":
            s = gpu_lib.Strips(nx, NY, 0.7, 1e-6, 0.0, mask, 3, precision=prec)
        else:
            s = gpu_lib.Solver(nx, NY, 0.7, 1e-6, 0.0, mask, precision=prec)
        with s:
            s.set_inflow_outflow(U)
            if isinstance(how, int):
                s.set_variant(how)
            s.set_populations(s0)
            if how == "single":
                for _ in range(STEPS):
                    s.step(1)
            else:
                s.run(STEPS)
            got.append(s.populations())
    for g in got[1:]:
        assert np.array_equal(g, got[0])
