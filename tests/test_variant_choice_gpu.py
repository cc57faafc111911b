"""The kernel that the automatic choice reports can be chosen (GPU): lbm_set_variant takes the number
that lbm_device_info gives after a run, and the run is the same; kernels of another storage form, or
that a grid does not fit, are refused. The block size in the report is the direct kernel's own, and
a block size that the caller sets is the one it runs."""
from __future__ import annotations

import re

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def report(s):
    info = s.bench_info()
    m = re.search(r'"block": "(\d+)x1".*_v(\d+)(_auto)?"', info)
    return int(m[1]), int(m[2]), m[3] is not None


@pytest.mark.parametrize("prec,nx,ny,steps,variant", [
    ("fp32", 300, 70, 20, 24), ("fp16", 300, 70, 20, 24), ("bf16", 517, 203, 9, 24), ("fp32", 300, 70, 3, 19),
    ("fp32", 2049, 1025, 6, 23), ("fp32", 8200, 5650, 2, 28), ("fp16", 2048, 2050, 6, 20), ("fp16", 4096, 2049, 6, 27),
    ("bf16", 4096, 2049, 6, 27), ("fp64", 512, 70, 20, 25), ("fp64", 300, 70, 20, 26)])
def test_the_reported_kernel_can_be_chosen(gpu_lib, prec, nx, ny, steps, variant):
    mask = gpu_lib.make_channel(nx, ny)
    got = []
    for choose in (False, True):
        with gpu_lib.Solver(nx, ny, 0.6, 1e-6, 0.0, mask, precision=prec) as s:
            if choose:
                s.set_variant(variant)
            s.init_equilibrium(1.0, 0.03, 0.01)
            s.run(steps)
            assert report(s)[1:] == (variant, not choose)
            got.append((s.macroscopic() if nx * ny > 1 << 24 else [s.populations()], s.total_mass()))
    assert got[0][1] == got[1][1]
    for a, b in zip(got[0][0], got[1][0]):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("prec,nx,ny,refused", [
    ("fp32", 64, 40, (25, 26, 27, 29, -2)), ("fp16", 64, 40, (23, 25, 26, 28, 29)), ("fp64", 64, 40, (23, 24, 27, 28, 29)),
    ("fp32", 2048, 1024, (24,)), ("bf16", 2048, 1024, (24,))])
def test_kernels_of_another_form_are_refused(gpu_lib, prec, nx, ny, refused):
    with gpu_lib.Solver(nx, ny, 0.6, 1e-6, 0.0, gpu_lib.make_channel(nx, ny), precision=prec) as s:
        for v in refused:
            with pytest.raises(ValueError):
                s.set_variant(v)


def test_block_size_of_the_fp64_direct_kernel(gpu_lib):
    nx, ny = 300, 70
    mask = gpu_lib.make_channel(nx, ny)
    got = []
    for block in (None, 256, 64, 0):
        with gpu_lib.Solver(nx, ny, 0.6, 1e-6, 0.0, mask, precision="fp64") as s:
            if block is not None:
                s.set_launch(block)
            s.init_equilibrium(1.0, 0.03, 0.01)
            s.run(5)
            assert report(s) == ({None: 128, 256: 256, 64: 64, 0: 128}[block], 26, True)
            got.append(s.populations())
    for g in got[1:]:
        assert np.array_equal(g, got[0])
