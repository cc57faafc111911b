"""The automatic 16-bit kernels of large grids (2048-cell tiles with 2 or 3 blocks per SM, 1024-cell
tiles where a row fills the wide ones badly) against the direct kernel, and the strips (GPU)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(2048, 2048), (4096, 2049), (3000, 1500), (2049, 2100), (3483, 1300)])
@pytest.mark.parametrize("form", ["fp16", "bf16"])
def test_large_16bit_kernels_agree(gpu_lib, nx, ny, form):
    mask = gpu_lib.geometry.add_block(gpu_lib.make_channel(nx, ny), nx, 1020, 1030, 90, 120)
    s0 = gpu_lib.workloads.seeded_state(9, 1e-3, nx, ny, mask, np.float32)
    got = []
    for variant in (-1, 0):
        with gpu_lib.Solver(nx, ny, 0.6, 1e-6, 0.0, mask, precision=form) as s:
            s.set_variant(variant)
            s.set_populations(s0)
            s.run(3)
            got.append(s.populations())
    with gpu_lib.Strips(nx, ny, 0.6, 1e-6, 0.0, mask, 3, precision=form) as h:
        h.set_populations(s0)
        h.run(3)
        got.append(h.populations())
    assert np.array_equal(got[0], got[1]) and np.array_equal(got[0], got[2])
