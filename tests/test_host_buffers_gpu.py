"""Host buffers of every kind give the same results (GPU): ordinary arrays, fresh anonymous memory
whose pages are not there yet (small and large), memory that is not aligned to its values (which
goes through device memory), pinned memory; and the strips' and ensembles' read back."""
from __future__ import annotations

import mmap

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def buffer(kind, count, dtype):
    size = count * np.dtype(dtype).itemsize
    if kind == "fresh":
        return np.frombuffer(mmap.mmap(-1, size), dtype=dtype, count=count)
    if kind == "misaligned":
        return np.frombuffer(mmap.mmap(-1, size + 8), dtype=dtype, count=count, offset=1)
    if kind == "offset":
        return np.frombuffer(mmap.mmap(-1, size + 64), dtype=dtype, count=count, offset=24)
    if kind == "pinned":
        import torch
        return torch.empty(count, dtype=torch.float64 if dtype == np.float64 else torch.float32,
                           pin_memory=True).numpy()
    return np.zeros(count, dtype)


@pytest.mark.parametrize("nx,ny", [(53, 31), (1021, 401), (2050, 1100)])
@pytest.mark.parametrize("prec", ["fp32", "fp64", "fp16"])
@pytest.mark.parametrize("kind", ["fresh", "misaligned", "offset", "pinned"])
def test_host_buffers_agree(gpu_lib, nx, ny, prec, kind):
    dt = np.float64 if prec == "fp64" else np.float32
    mask = gpu_lib.geometry.add_block(gpu_lib.make_channel(nx, ny), nx, 12, 16, 10, 17)
    s0 = gpu_lib.workloads.seeded_state(4, 1e-3, nx, ny, mask, dt)
    n = nx * ny
    with gpu_lib.Solver(nx, ny, 0.7, 1e-6, 0.0, mask, precision=prec) as s:
        src = buffer(kind, 9 * n, dt)
        src[:] = s0
        assert gpu_lib.lib().lbm_set_populations(s.handle, gpu_lib._ptr(src)) == gpu_lib.OK
        s.run(5)
        got = [s.populations(out=buffer(kind, 9 * n, dt)), *s.macroscopic(out=[buffer(kind, n, dt) for _ in range(3)])]
        point, mass, finite = s.populations_at(20, 20), s.total_mass(), s.check_finite()
        s.set_populations(s0)  # another run of the same: the 16-bit forms' rounding moves on
        s.run(5)
        again = s.populations()
    with gpu_lib.Solver(nx, ny, 0.7, 1e-6, 0.0, mask, precision=prec) as s:
        s.set_populations(np.array(s0))
        s.run(5)
        want = [s.populations(), *s.macroscopic()]
        assert finite and s.check_finite() and mass == s.total_mass()
        assert np.array_equal(point, s.populations_at(20, 20))
    for a, b in zip(got, want):
        assert np.array_equal(a, b)
    if prec != "fp16":
        assert np.array_equal(again, want[0])
    assert np.array_equal(point, want[0].reshape(ny, nx, 9)[20, 20])


@pytest.mark.parametrize("strips", [1, 4])
def test_strips_and_batch_read_back(gpu_lib, strips):
    nx, ny = 517, 203
    mask = gpu_lib.geometry.add_block(gpu_lib.make_channel(nx, ny), nx, 12, 16, 10, 17)
    s0 = gpu_lib.workloads.seeded_state(4, 1e-3, nx, ny, mask, np.float32)
    spec = {"nx": nx, "ny": ny, "mask": mask, "tau": 0.7, "fx": 1e-6}
    with gpu_lib.Solver(nx, ny, 0.7, 1e-6, 0.0, mask) as s, gpu_lib.Strips(nx, ny, 0.7, 1e-6, 0.0, mask, strips) as h, \
            gpu_lib.Batch([spec], precision="fp32") as b:
        s.set_populations(s0)
        h.set_populations(s0)
        b.set_populations(0, s0)
        for x in (s, h, b):
            x.run(3)
        want = s.populations()
        assert np.array_equal(h.populations(), want) and np.array_equal(b.populations(0), want)
        for a, c in zip(h.macroscopic(), s.macroscopic()):
            assert np.array_equal(a, c)
