"""What a backward run may take from the forward run before it (GPU): a drag field taken away in between
makes it compute its states anew, and a forward run whose checkpoints find no memory leaves nothing to
go back over or to read."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("every", [40, 100])
def test_field_removed_after_the_forward_run(gpu_lib, prec, every):
    nx, ny, steps, window = 130, 24, 30, 7
    mask = gpu_lib.make_channel(nx, ny)
    alpha = np.linspace(0.0, 0.1, nx * ny)
    with gpu_lib.Adjoint(nx, ny, 0.7, 1e-5, 0.0, mask, precision=prec, checkpoint_every=every) as a, \
            gpu_lib.Adjoint(nx, ny, 0.7, 1e-5, 0.0, mask, precision=prec, checkpoint_every=every) as plain:
        a.set_alpha(alpha)
        a.forward(steps, window)
        a.backward()
        a.forward(steps, window)  # its states stay for the backward run
        a.set_alpha(None)
        got = a.backward()
        plain.forward(steps, window)
        want = plain.backward()
    for k in ("tau", "fx", "fy", "alpha"):
        assert np.array_equal(got[k], want[k]), k


def test_forward_run_without_memory_for_its_checkpoints(gpu_lib):
    nx, ny = 130, 24
    mask = gpu_lib.make_channel(nx, ny)
    with gpu_lib.Adjoint(nx, ny, 0.7, 1e-5, 0.0, mask, precision="fp32", checkpoint_every=1) as a:
        j = a.forward(6, 2)
        g = a.backward()
        with pytest.raises(gpu_lib.LbmError) as e:
            a.forward(2_000_000_000, 1)  # hundreds of terabytes: refused at once
        assert e.value.code == gpu_lib.ERR_OUT_OF_MEMORY
        with pytest.raises(ValueError):
            a.backward()
        with pytest.raises(ValueError):
            a.populations()
        assert np.array_equal(a.forward(6, 2), j)
        assert np.array_equal(a.backward()["alpha"], g["alpha"])
