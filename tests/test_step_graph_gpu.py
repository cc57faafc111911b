"""Long runs of the step kernels replay CUDA graphs of 32 launches (GPU): the same bits as single
launches, with the 16-bit forms' rounding keys read from the device's step counter, also where
resident launches and single steps alternate with them. A block size of 128 keeps a small grid on
the step kernels."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["fp32", "fp64", "fp16", "bf16"])
@pytest.mark.parametrize("nx,ny,open_x", [(300, 70, False), (300, 70, True), (130, 41, False), (2049, 40, False)])
def test_graph_replay_equals_single_launches(gpu_lib, form, nx, ny, open_x):
    mask = gpu_lib.workloads.cylinder_wake(nx, ny, d=12.0, xc=60.0, yc=ny / 2)
    with gpu_lib.Solver(nx, ny, 0.56, 2e-6, 0.0, mask, precision=form) as a, \
            gpu_lib.Solver(nx, ny, 0.56, 2e-6, 0.0, mask, precision=form) as b, \
            gpu_lib.Solver(nx, ny, 0.56, 2e-6, 0.0, mask, precision=form) as c:
        for s in (a, b, c):
            if open_x:
                s.set_inflow_outflow(0.03)
            s.init_equilibrium(1.0, 0.03, 0.0)
        a.set_launch(128)
        b.set_launch(128)
        a.run(203)  # graphs of 32 launches, then single launches
        a.run(64)   # graphs from the other buffer
        for _ in range(267):
            b.step(1)
        for n in (1, 100, 3, 2, 33, 128):  # resident where the form and the grid allow, and single steps
            c.run(n)
        assert np.array_equal(a.populations(), b.populations())
        assert np.array_equal(c.populations(), b.populations())
