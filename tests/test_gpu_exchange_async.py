"""eb_step_host_state with inputs and no outputs (GPU): it returns once the
inputs are the caller's again, before the steps have run."""
import time

import numpy as np
import pytest

import elasticapp_b200 as eb
from elasticapp_b200 import workloads as W

pytestmark = pytest.mark.gpu


def test_inputs_alone_do_not_wait_for_the_steps():
    import torch

    wl = W.uneven_batch(n_rods=4096, seed=5)
    sim = wl.build(step_mode="streaming")
    v = torch.zeros((3, sim.n_slots()), dtype=torch.float64, pin_memory=True).numpy()
    want = np.random.default_rng(6).normal(0.0, 1e-3, v.shape)
    t = sim.step_host_state(eb.PositionVerlet(), 0.0, wl.dt, 4, inputs={"Velocity": v})
    sim.synchronize()
    state = {n: sim.get_slots(n) for n in ("Position", "Velocity", "Director", "AngularVelocity")}
    v[:] = want
    t0 = time.perf_counter()
    sim.step_host_state(eb.PositionVerlet(), t, wl.dt, 300, inputs={"Velocity": v})
    t1 = time.perf_counter()
    v[:] = np.nan  # the caller's again
    sim.synchronize()
    t2 = time.perf_counter()
    assert t1 - t0 < 0.5 * (t2 - t0), (t1 - t0, t2 - t0)
    got = sim.get_slots("Position")
    for n in state:
        sim.set_slots(n, want if n == "Velocity" else state[n])
    sim.step(eb.PositionVerlet(), t, wl.dt, 300)
    np.testing.assert_array_equal(got, sim.get_slots("Position"))
    sim.close()
