"""Strips read back into memory that takes a copy (GPU): the staging buffer holds one strip, not the
lattice, so that a lattice which nearly fills the device can still be read; the values are those
of an ordinary array."""
from __future__ import annotations

import mmap

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def misaligned(count, dtype):
    return np.frombuffer(mmap.mmap(-1, count * np.dtype(dtype).itemsize + 8), dtype=dtype, count=count, offset=1)


@pytest.mark.parametrize("prec", ["fp32", "fp64", "fp16"])
@pytest.mark.parametrize("strips", [1, 8, 17])
def test_read_back_stages_one_strip(gpu_lib, prec, strips):
    import torch
    nx, ny = 1030, 1025
    n = nx * ny
    dt = np.float64 if prec == "fp64" else np.float32
    mask = gpu_lib.geometry.add_block(gpu_lib.make_channel(nx, ny), nx, 250, 262, 90, 120)
    s0 = gpu_lib.workloads.seeded_state(9, 1e-3, nx, ny, mask, dt)
    lib = gpu_lib.lib()
    with gpu_lib.Strips(nx, ny, 0.6, 1e-6, 0.0, mask, strips, precision=prec) as h:
        h.set_populations(s0)
        h.run(3)
        want = [h.populations(), *h.macroscopic()]
        pops, fields = misaligned(9 * n, dt), [misaligned(n, dt) for _ in range(3)]
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        assert lib.lbm_strips_get_populations(h._h, gpu_lib._ptr(pops)) == gpu_lib.OK
        assert lib.lbm_strips_macroscopic(h._h, *map(gpu_lib._ptr, fields)) == gpu_lib.OK
        # The upload's staging buffer holds a strip and its ghost rows already (2 MB: the
        # allocator's grain).
        assert free - torch.cuda.mem_get_info()[0] <= (2 << 20)
    for a, b in zip([pops, *fields], want):
        assert np.array_equal(a, b)
