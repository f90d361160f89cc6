"""Streaming steps whose launches overlap the ones before them, interleaved
with changes of the state and the parameters (GPU)."""
import numpy as np
import pytest

import elasticapp_b200 as eb
from elasticapp_b200 import workloads as W

pytestmark = pytest.mark.gpu

STATE = (("Position", 0), ("Velocity", 0), ("Director", 1), ("AngularVelocity", 1))


@pytest.mark.parametrize("rods", [3, 700])
def test_changes_between_steps_reach_the_next_launch(rods):
    # single steps in quick succession against the same steps with the device
    # idle between them: a launch must see every copy made before it
    wl = W.uneven_batch(n_rods=rods, seed=32, n_range=(20, 300))
    out = []
    for wait in (False, True):
        sim = wl.build(step_mode="streaming")
        rng, t = np.random.default_rng(33), 0.0
        for k in range(12):
            t = sim.step(eb.PositionVerlet(), t, wl.dt * (1 + (k % 3 == 2)), 1)  # (another dt: another damper table)
            if wait:
                sim.synchronize()
            if k % 4 == 1:
                sim.set_slots("Velocity", sim.get_slots("Velocity") + rng.normal(0, 1e-3, (3, sim.n_slots())))
            if k % 4 == 3:
                sim.set_slots("Mass", sim.get_slots("Mass") * 1.5)
        out.append({name: sim.get_slots(name) for name, _ in STATE})
        sim.close()
    for name, _ in STATE:
        assert np.array_equal(out[0][name], out[1][name]), name
