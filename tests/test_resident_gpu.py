"""Resident launches (the state in shared memory over many steps) against one launch per step, on
the GPU: the same bits for every storage form, at the edges of the tiles and of what fits. The
per-step kernels are selected with set_launch(128) and are pinned to the reference elsewhere."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GRIDS = [(1, 7), (2, 3), (3, 1), (33, 65), (64, 1), (65, 305), (128, 66), (129, 152), (300, 700), (1021, 301),
         (1025, 257), (1987, 150)]


def channel(pkg, nx, ny):
    if ny < 3 or nx < 16:
        mask = np.zeros((ny, nx), np.uint8)
        if nx * ny > 4:
            mask[0, 0] = 1
        return mask.reshape(-1)
    mask = pkg.make_channel(nx, ny).reshape(ny, nx).copy()
    for x, y in ((nx // 3, ny // 2), (nx - 1, ny // 3), (0, ny // 4), (32 % nx, ny // 2), (nx // 2, 1)):
        mask[y, x] = 1
    return mask.reshape(-1)


@pytest.mark.parametrize("nx,ny", GRIDS)
@pytest.mark.parametrize("form", ["fp32", "fp16", "bf16"])
@pytest.mark.parametrize("open_x", [False, True])
def test_resident_equals_per_step(gpu_lib, nx, ny, form, open_x):
    if open_x and nx < 3:
        pytest.skip("open boundaries need nx >= 3")
    mask = channel(gpu_lib, nx, ny)
    if open_x:  # the outlet columns stay fluid
        m = mask.reshape(ny, nx).copy()
        m[1:-1, -2:] = 0
        mask = m.reshape(-1)
    out = []
    for resident in (True, False):
        with gpu_lib.Solver(nx, ny, 0.62, 1e-6, 2e-7 if nx % 2 else 0.0, mask, precision=form) as s:
            if open_x:
                s.set_inflow_outflow(0.04)
            s.init_equilibrium(1.0, 0.04, 0.0)
            if not resident:
                s.set_launch(128)
            s.run(5)
            s.run(38)  # an odd and an even number of steps, two launches
            out.append((s.populations(), *s.macroscopic()))
    for a, b in zip(*out):
        assert np.array_equal(a, b)


def test_resident_in_a_captured_graph(gpu_lib):
    """Replays of a captured run carry on from the device's step counter."""
    import torch
    nx, ny = 200, 96
    mask = channel(gpu_lib, nx, ny)
    with gpu_lib.Solver(nx, ny, 0.6, 1e-6, 0.0, mask, precision="fp16") as a, \
            gpu_lib.Solver(nx, ny, 0.6, 1e-6, 0.0, mask, precision="fp16") as b:
        for s in (a, b):
            s.init_equilibrium(1.0, 0.03, 0.0)
        stream = torch.cuda.Stream()
        a.set_stream(stream.cuda_stream)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            a.step(6)
        for _ in range(5):
            graph.replay()
        torch.cuda.synchronize()
        for _ in range(30):
            b.step(1)
        assert np.array_equal(a.populations(), b.populations())


def test_two_resident_solvers_on_two_streams(gpu_lib):
    nx, ny = 512, 200
    mask = channel(gpu_lib, nx, ny)
    got = []
    with gpu_lib.Solver(nx, ny, 0.6, 1e-6, 0.0, mask) as a, gpu_lib.Solver(nx, ny, 0.6, 1e-6, 0.0, mask) as b:
        for s in (a, b):
            s.init_equilibrium(1.0, 0.03, 0.0)
        for _ in range(20):
            a.step(7)
            b.step(7)
        got = [a.populations(), b.populations()]
    assert np.array_equal(*got)


def ensemble(pkg, count, lo, hi, fy):
    specs = []
    r = np.random.RandomState(count)
    for k in range(count):
        nx, ny = int(r.randint(lo, hi)), int(r.randint(3, hi // 2))
        specs.append({"nx": nx, "ny": ny, "mask": channel(pkg, nx, ny), "tau": 0.55 + 0.4 * r.rand(),
                      "fx": 1e-6 * k, "fy": fy})
    return specs


@pytest.mark.parametrize("count,lo,hi", [(1, 65, 66), (5, 3, 40), (24, 30, 200), (40, 64, 130), (152, 3, 33)])
@pytest.mark.parametrize("form", ["fp32", "fp16", "bf16"])
def test_resident_ensemble_equals_separate(gpu_lib, count, lo, hi, form):
    """A small ensemble's resident launches against one launch per instance and step, with an
    autotuning in between (it puts the step counter back: resident states keep their numbers)."""
    specs = ensemble(gpu_lib, count, lo, hi, 3e-7 if count == 24 else 0.0)
    got = []
    for resident in (True, False):
        with gpu_lib.Batch(specs, precision=form) as b:
            b.init_equilibrium(1.0, 0.03, 0.01)
            for n in (9, 4, 22):
                if resident:
                    b.run(n)
                    if n == 9 and count == 5:
                        b.autotune()
                else:
                    b.run_separate(n)
            got.append([b.populations(k) for k in range(count)])
    for a, c in zip(*got):
        assert np.array_equal(a, c)
