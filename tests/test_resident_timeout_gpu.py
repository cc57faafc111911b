"""The failure path of resident launches (GPU): a block's wait for its neighbours' words, made to run
out on purpose. lbm_test_set_consumer_wait_limit(1) ends a wait whose word is not there at the first
look; every block then leaves its steps and ends, so no wait goes on. The call reports
LBM_ERR_TIMEOUT and clears the flag, and after the state is set again a normal run is right: the
numbers of the states went on, so no word of the failed launch passes for a later one."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NX, NY = 517, 203


@pytest.fixture
def short_waits(gpu_lib):
    lib = gpu_lib.lib()
    assert lib.lbm_test_set_consumer_wait_limit(1) == gpu_lib.OK

    def restore():
        assert lib.lbm_test_set_consumer_wait_limit(0) == gpu_lib.OK
    yield restore
    restore()


@pytest.mark.parametrize("form", ["fp32", "fp16"])
@pytest.mark.parametrize("open_x", [False, True])
@pytest.mark.parametrize("steps", [40, 8200])
def test_solver(gpu_lib, short_waits, form, open_x, steps):
    lib = gpu_lib.lib()
    mask = gpu_lib.geometry.add_block(gpu_lib.make_channel(NX, NY), NX, 12, 16, 10, 17)
    args = (NX, NY, 0.6, 1e-6, 0.0, mask)
    s0 = gpu_lib.workloads.seeded_state(4, 1e-3, NX, NY, mask, np.float32)
    with gpu_lib.Solver(*args, precision=form) as s, gpu_lib.Solver(*args, precision=form) as want:
        for x in (s, want):
            if open_x:
                x.set_inflow_outflow(0.04)
            x.set_populations(s0)
        assert lib.lbm_run(s.handle, steps) == gpu_lib.ERR_TIMEOUT
        assert "gave up waiting" in lib.lbm_last_error(s.handle).decode()
        assert lib.lbm_synchronize(s.handle) == gpu_lib.OK  # the flag was cleared
        assert '_v24_auto"' in s.bench_info()
        short_waits()
        want.set_launch(128)
        if form == "fp16":  # the rounding keys go on with the steps
            for _ in range(steps // 8):
                want.step(8)
            want.step(steps % 8)
        for x in (s, want):
            x.set_populations(s0)
            x.run(21)
        assert np.array_equal(s.populations(), want.populations())


@pytest.mark.parametrize("form", ["fp32", "bf16"])
def test_ensemble(gpu_lib, short_waits, form):
    specs = []
    for k in range(9):
        nx, ny = 64 + 23 * k, 40 + 7 * k
        specs.append({"nx": nx, "ny": ny, "mask": gpu_lib.make_channel(nx, ny), "tau": 0.6, "fx": 1e-6 * k, "fy": 0.0})
    with gpu_lib.Batch(specs, precision=form) as b, gpu_lib.Batch(specs, precision=form) as want:
        b.init_equilibrium(1.0, 0.03, 0.01)
        with pytest.raises(gpu_lib.LbmError) as e:
            b.run(40)
        assert e.value.code == gpu_lib.ERR_TIMEOUT and "gave up waiting" in str(e.value)
        short_waits()
        want.init_equilibrium(1.0, 0.03, 0.01)
        want.run_separate(40)
        for x in (b, want):
            x.init_equilibrium(1.0, 0.03, 0.01)
        b.run(21)
        want.run_separate(21)
        for k in range(len(specs)):
            assert np.array_equal(b.populations(k), want.populations(k))
