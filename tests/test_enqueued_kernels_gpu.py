"""lbm_enqueued_kernels counts the kernels that a run really enqueues (GPU): resident, graph-replayed
and direct runs, with and without the 16-bit forms' step-counter updates; a captured run's count is
the number of the graph's kernel nodes."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


def counts(pkg, form, runs, launch=None, nx=300):
    mask = pkg.make_channel(nx, 70)
    got = []
    with pkg.Solver(nx, 70, 0.6, 1e-6, 0.0, mask, precision=form) as s:
        if launch:
            s.set_launch(launch)
        s.init_equilibrium(1.0, 0.0, 0.0)
        for n in runs:
            k = s.enqueued_kernels()
            s.run(n)
            got.append(s.enqueued_kernels() - k)
    return got


@pytest.mark.parametrize("form", ["fp32", "fp16", "bf16"])
def test_resident(gpu_lib, form):
    # One launch and one counter update for at most 8192 steps; fewer than four steps are not resident.
    update = form != "fp32"
    assert counts(gpu_lib, form, [4, 5, 200, 8192, 8193, 20000, 3, 1]) == [2, 2, 2, 2, 4, 6, 3 + update, 1 + update]


@pytest.mark.parametrize("form", ["fp32", "fp64", "fp16"])
def test_step_kernels(gpu_lib, form):
    update = form == "fp16"
    # 6 graphs of 32 steps and 8 direct steps; direct steps alone; one graph alone.
    want = [200 + 7 * update, 5 + update, 32 + update, 31 + update]
    assert counts(gpu_lib, form, [200, 5, 32, 31], launch=128) == want


@pytest.mark.parametrize("form", ["fp32", "fp16"])
@pytest.mark.parametrize("launch,steps", [(None, 6), (128, 6), (None, 9000)])
def test_captured_run_has_as_many_kernel_nodes(gpu_lib, form, launch, steps):
    import ctypes
    import torch
    mask = gpu_lib.make_channel(300, 70)
    rt = ctypes.CDLL(None)  # the CUDA runtime that torch has loaded
    if not hasattr(rt, "cudaGraphGetNodes"):
        rt = next((ctypes.CDLL(line.split()[-1]) for line in open("/proc/self/maps") if "libcudart" in line), None)
    if rt is None:
        pytest.skip("the CUDA runtime library is not to be found")
    with gpu_lib.Solver(300, 70, 0.6, 1e-6, 0.0, mask, precision=form) as s:
        stream = torch.cuda.Stream()
        s.set_stream(stream.cuda_stream)
        if launch:
            s.set_launch(launch)
        s.init_equilibrium(1.0, 0.0, 0.0)
        s.synchronize()
        handle = ctypes.c_void_p(stream.cuda_stream)
        graph, count = ctypes.c_void_p(), ctypes.c_size_t()
        k = s.enqueued_kernels()
        assert rt.cudaStreamBeginCapture(handle, 2) == 0
        s.step(steps)
        assert rt.cudaStreamEndCapture(handle, ctypes.byref(graph)) == 0
        assert rt.cudaGraphGetNodes(graph, None, ctypes.byref(count)) == 0
        assert count.value == s.enqueued_kernels() - k
        assert rt.cudaGraphDestroy(graph) == 0
