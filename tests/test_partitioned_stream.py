"""A stream on a partition of the SMs (a green context): resident launches need a block on every SM
of their cut at once, so such a stream takes the step kernels. The SM count is told on the host
against a stand-in for the driver; the runs themselves on the GPU."""
from __future__ import annotations

import ctypes
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]


def cuda_include():
    return Path(shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc").resolve().parents[1] / "include"


@pytest.mark.parametrize("driver", ["known", "unknown"])
def test_stream_sm_count(tmp_path, driver):
    if shutil.which("g++") is None or not (cuda_include() / "cuda.h").exists():
        pytest.skip("no host compiler or CUDA headers")
    exe = tmp_path / "stream_sms_test"
    pkgdir = next(ROOT.glob("simulation-de-fluide-*_gb300"))
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(pkgdir / "csrc"), "-I", str(cuda_include()),
                    str(ROOT / "tests" / "cpp" / "stream_sms_test.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe), driver], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.gpu
@pytest.mark.parametrize("prec", ["fp32", "fp16"])
def test_a_stream_on_some_of_the_sms(gpu_lib, tmp_path, prec):
    import torch
    torch.zeros(1, device="cuda")  # the primary context is current
    so = tmp_path / "green_stream.so"
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", str(cuda_include()),
                    str(ROOT / "tests" / "cpp" / "green_stream.cpp"), "-ldl", "-o", str(so)], check=True)
    green = ctypes.CDLL(str(so))
    stream, ctx, got = ctypes.c_void_p(), ctypes.c_void_p(), ctypes.c_uint()
    rc = green.green_stream_create(16, ctypes.byref(stream), ctypes.byref(ctx), ctypes.byref(got))
    if rc != 0:
        pytest.skip(f"no SM partitions here ({rc})")
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert 0 < got.value < sms
    nx, ny, steps = 512, 200, 40
    mask = gpu_lib.make_channel(nx, ny)
    out, info = [], []
    try:
        for partitioned in (False, True):
            with gpu_lib.Solver(nx, ny, 0.6, 1e-6, 0.0, mask, precision=prec) as s:
                if partitioned:
                    s.set_stream(stream.value)
                s.init_equilibrium(1.0, 0.03, 0.0)
                s.run(steps)
                info.append(s.bench_info())
                out.append(s.populations())
    finally:
        green.green_stream_destroy(stream, ctx)
    assert '_v24_auto"' in info[0] and '_v24_auto"' not in info[1]
    assert np.array_equal(*out)
