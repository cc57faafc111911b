"""What a backward run may take from the forward run before it (GPU): a drag field taken away in between
makes it compute its states anew."""
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
