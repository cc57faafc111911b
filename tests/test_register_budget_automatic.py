"""Register budgets of the kernels that the automatic choices launch, beside those of
test_register_budget.py: the FP32 rings of large grids, the resident kernels of every force kind, the
kernels with FP64 products on the integer units, the strip engine's and the wide adjoint sweeps
(CPU only, needs nvcc). Each keeps the warps it is sized for on an SM, and spills no more than
stated: nothing, but a few words in the open 16-bit forms with four passes, and 200 to 400 bytes in
FP64 with integer products, whose three blocks per SM at 72 registers beat one block without a
spill (4.73k against 4.17k MLUPS at 1024 x 512)."""
from __future__ import annotations

import shutil
import sys
import tempfile
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

import pytest

import test_register_budget as budget

_compiled = {}


def _report_once(unit, *args, _report=budget.ptxas_report):
    """A translation unit is compiled once for both modules (minutes each)."""
    if unit not in _compiled:
        _compiled[unit] = _report(unit, *args)
    return _compiled[unit]


budget.ptxas_report = _report_once

F32, INT = "float, ExactPhys<ExactF32>", "double, ExactPhys<ExactF64Int>"
H16 = ["__half, FastPhys", "__nv_bfloat16, FastPhys"]

# (translation unit, kernel, warps per block, resident blocks per SM, most bytes of spill stores)
KERNELS = [("solver.cu", f"ring_step_kernel<{F32}, 0, 4, 2, 2, 5>", 5, 5, 0),
           ("solver.cu", f"ring_step_kernel<{F32}, 1, 4, 2, 2, 5>", 5, 5, 0),
           ("solver.cu", f"ring_step_kernel<{F32}, 0, 4, 2, 3, 1>", 5, 3, 0),
           ("solver.cu", f"ring_step_kernel<{F32}, 1, 4, 2, 3, 1>", 5, 3, 0),
           ("solver.cu", f"ring_step_kernel<{F32}, 0, 8, 2, 2, 3>", 9, 3, 0),
           ("solver.cu", f"ring_step_kernel<{F32}, 0, 8, 1, 4, 3>", 9, 3, 0),
           ("batch.cu", f"batch_ring_kernel<{INT}, 4, 2, 2>", 5, 4, 400),
           ("strips.cu", f"strip_ring_kernel<{F32}, 0, 4, 2, 5>", 5, 5, 0),
           ("strips.cu", f"strip_ring_kernel<{F32}, 0, 8, 2, 3>", 9, 3, 0),
           ("adjoint.cu", "adj_backward_kernel<float, 2, 2, 2>", 9, 2, 0),
           ("adjoint.cu", "adj_forward_kernel<ExactF64Int, 1, 3, 3>", 9, 3, 256),
           ("adjoint.cu", "adj_backward_kernel<double, 1, 2, 2>", 9, 2, 0)]
for open_x in (0, 1):
    KERNELS += [("solver.cu", f"pull_step_kernel<{INT}, {open_x}, 0>", 4, 3, 0),
                ("solver.cu", f"ring_step_kernel<{INT}, {open_x}, 8, 1, 4, 3>", 9, 3, 256),
                ("strips.cu", f"strip_ring_kernel<{INT}, {open_x}, 8, 1, 3>", 9, 3, 272)]
    for kind in (0, 1, 2):
        KERNELS += [("solver.cu", f"resident_step_kernel<{F32}, {open_x}, {kind}>", 32, 1, 0)]
        KERNELS += [("solver.cu", f"resident_step_kernel<{h}, {open_x}, {kind}>", 28, 1, 0) for h in H16]
    for h in H16:
        KERNELS += [("solver.cu", f"ring_step_kernel<{h}, {open_x}, 8, 4, 2, 2>", 9, 2, 8 * open_x),
                    ("solver.cu", f"ring_step_kernel<{h}, {open_x}, 8, 2, 2, 3>", 9, 3, 0),
                    ("solver.cu", f"ring_step_kernel<{h}, {open_x}, 8, 1, 4, 3>", 9, 3, 0),
                    ("strips.cu", f"strip_ring_kernel<{h}, {open_x}, 8, 2, 3>", 9, 3, 0),
                    ("strips.cu", f"strip_ring_kernel<{h}, {open_x}, 8, 4, {3 - open_x}>", 9, 3 - open_x, 56 * open_x)]
for kind in (0, 1, 2):
    KERNELS += [("batch.cu", f"batch_resident_kernel<{F32}, {kind}>", 32, 1, 0)]
    KERNELS += [("batch.cu", f"batch_resident_kernel<{h}, {kind}>", 28, 1, 0) for h in H16]


@pytest.fixture(scope="module")
def reports():
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    filt = shutil.which("cu++filt") or "/usr/local/cuda/bin/cu++filt"
    if not Path(nvcc).exists() or not Path(filt).exists():
        pytest.skip("nvcc / cu++filt not available")
    sys.path.insert(0, str(budget.PKG))
    import buildlib
    units = sorted({u for u, *_ in KERNELS})
    with tempfile.TemporaryDirectory() as d, ThreadPoolExecutor(len(units)) as ex:
        futs = {u: ex.submit(budget.ptxas_report, u, buildlib.common_flags, nvcc, filt, d) for u in units}
        return {u: f.result() for u, f in futs.items()}


@pytest.mark.parametrize("unit,kernel,warps,blocks,spilled", KERNELS)
def test_automatic_kernel_fits_its_register_budget(reports, unit, kernel, warps, blocks, spilled):
    assert kernel in reports[unit], f"kernel {kernel} not compiled in {unit}"
    regs, spill = reports[unit][kernel]
    assert spill <= spilled, f"{kernel}: {spill} bytes of spill stores"
    per_warp = (regs + 7) // 8 * 8 * 32
    assert -(-warps * blocks // 4) * per_warp <= 16384, f"{kernel}: {regs} registers, fewer than {blocks} blocks of {warps} warps"
