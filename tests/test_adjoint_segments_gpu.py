"""The adjoint's last segment kept from the forward run (GPU): gradients, final state and
objectives of repeated forward / backward calls on one object equal those of a fresh object,
where the last segment is whole, short, one step long, or the only one."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("steps,every", [(12, 4), (13, 4), (9, 4), (7, 10), (10, 10), (1, 3), (5, 1)])
def test_repeated_runs_equal_fresh_ones(gpu_lib, prec, steps, every):
    nx, ny, batch = 300, 24, 3
    mask = gpu_lib.geometry.add_block(gpu_lib.make_channel(nx, ny), nx, 250, 262, 9, 14)
    fields = [gpu_lib.workloads.brinkman_batch(nx, ny, batch, mask, seed=s) for s in (5, 50)]

    def fresh(alpha):
        with gpu_lib.Adjoint(nx, ny, 0.7, 1e-5, 1e-6, mask, precision=prec, batch=batch, checkpoint_every=every) as a:
            a.set_alpha(alpha)
            j = a.forward(steps, min(3, steps))
            return j, a.backward(), a.populations(1)

    want = [fresh(f) for f in fields]
    with gpu_lib.Adjoint(nx, ny, 0.7, 1e-5, 1e-6, mask, precision=prec, batch=batch, checkpoint_every=every) as a:
        for k in (0, 1, 1, 0):
            a.set_alpha(fields[k])
            j = a.forward(steps, min(3, steps))
            before = a.populations(1)
            g = [a.backward(), a.backward()]  # the second run cannot rely on what the first left
            assert np.array_equal(j, want[k][0])
            for r in g:
                for key in ("tau", "fx", "fy", "alpha"):
                    assert np.array_equal(r[key], want[k][1][key]), (k, key)
            assert np.array_equal(before, want[k][2]) and np.array_equal(a.populations(1), want[k][2])
