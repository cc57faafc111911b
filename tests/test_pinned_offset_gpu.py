"""Pinned host memory at any byte offset (GPU): where the values are not aligned the buffer takes a
copy, and every upload and read back gives the values of ordinary arrays."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def pinned_at(count, dtype, offset):
    import torch
    raw = torch.empty(count * np.dtype(dtype).itemsize + 64, dtype=torch.uint8, pin_memory=True).numpy()
    return np.frombuffer(raw.data, dtype=dtype, count=count, offset=offset)


@pytest.mark.parametrize("offset", [0, 1, 2, 4, 8, 12])
@pytest.mark.parametrize("prec", ["fp32", "fp64", "fp16"])
def test_every_engine_takes_pinned_memory_at_any_offset(gpu_lib, prec, offset):
    nx, ny = 131, 40
    n = nx * ny
    dt = np.float64 if prec == "fp64" else np.float32
    mask = gpu_lib.geometry.add_block(gpu_lib.make_channel(nx, ny), nx, 30, 41, 9, 17)
    s0 = gpu_lib.workloads.seeded_state(7, 1e-3, nx, ny, mask, dt)
    src = pinned_at(9 * n, dt, offset)
    src[:] = s0
    args = (nx, ny, 0.7, 1e-6, 0.0, mask)
    spec = {"nx": nx, "ny": ny, "mask": mask, "tau": 0.7, "fx": 1e-6}
    with gpu_lib.Solver(*args, precision=prec) as s, gpu_lib.Strips(*args, 3, precision=prec) as h, \
            gpu_lib.Batch([spec], precision=prec) as b:
        assert gpu_lib.lib().lbm_set_populations(s.handle, gpu_lib._ptr(src)) == gpu_lib.OK
        h.set_populations(s0)
        b.set_populations(0, src)
        fields = s.macroscopic()
        for a, w in zip(s.macroscopic(out=[pinned_at(n, dt, offset) for _ in range(3)]), fields):
            assert np.array_equal(a, w)
        want = s.populations()
        assert np.array_equal(s.populations(out=pinned_at(9 * n, dt, offset)), want)
        lib = gpu_lib.lib()
        for call, handle in ((lib.lbm_strips_get_populations, (h._h,)), (lib.lbm_batch_get_populations, (b._h, 0))):
            out = pinned_at(9 * n, dt, offset)
            assert call(*handle, gpu_lib._ptr(out)) == gpu_lib.OK
            assert np.array_equal(out, want)


@pytest.mark.parametrize("offset", [0, 1, 4, 8])
@pytest.mark.parametrize("prec", ["fp32", "fp64"])
def test_adjoint_takes_pinned_memory_at_any_offset(gpu_lib, prec, offset):
    nx, ny = 70, 24
    n = nx * ny
    dt = np.float64 if prec == "fp64" else np.float32
    mask = gpu_lib.make_channel(nx, ny)
    alpha = pinned_at(n, np.float64, offset)
    alpha[:] = np.linspace(0.0, 0.2, n)
    lib = gpu_lib.lib()
    got = []
    for field, grad, pops in ((np.array(alpha), np.empty(n), np.empty(9 * n, dt)),
                              (alpha, pinned_at(n, np.float64, offset), pinned_at(9 * n, dt, offset))):
        with gpu_lib.Adjoint(nx, ny, 0.7, 1e-5, 0.0, mask, precision=prec, checkpoint_every=4) as a:
            assert lib.lbm_adj_set_alpha(a._h, gpu_lib._ptr(field)) == gpu_lib.OK
            a.forward(9, 3)
            one = np.zeros(3)
            assert lib.lbm_adj_backward(a._h, *(gpu_lib._ptr(one[k:]) for k in range(3)), gpu_lib._ptr(grad)) == gpu_lib.OK
            assert lib.lbm_adj_get_populations(a._h, 0, gpu_lib._ptr(pops)) == gpu_lib.OK
            got.append((grad.copy(), pops.copy()))
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1])
