"""Resident FP64 kernel: the register and the looped form agree bit for bit on
states that stay finite (GPU), at rotations below the guarded range, small, and
past the small-angle series (0.2 rad a half step)."""
import numpy as np
import pytest

import elasticapp_b200 as eb
from elasticapp_b200 import workloads as W

pytestmark = pytest.mark.gpu

FIELDS = ("Position", "Velocity", "Director", "AngularVelocity")


@pytest.mark.parametrize("stepper", [eb.PositionVerlet, eb.VelocityVerlet, eb.PEFRL])
@pytest.mark.parametrize("omega,steps", [(0.0, 9), (1e-9, 9), (3.0, 9), (4e6, 1)])
def test_forms_agree_on_finite_states(stepper, omega, steps):
    lengths = (2, 3, 263, 255, 256, 7)
    wl = W.uneven_batch(n_rods=len(lengths), seed=11, n_range=(2, 2))
    for rod, n in zip(wl.rods, lengths):
        rod.n_elements = n
    wl.velocities = [np.random.default_rng(12 + n).normal(0.0, 1e-3, size=(3, n + 1)) for n in lengths]
    states = []
    for config in (1, 2, 3, 4):  # 520 slots on 512 and on 256 threads, 264 on 256, 320 on 320
        sim = wl.build(resident_config=config, step_mode="resident", stepper=stepper)
        sim.set_slots("AngularVelocity", np.random.default_rng(3).uniform(-1.0, 1.0, (3, sim.n_slots())) * omega)
        sim.step(stepper(), 0.0, 1e-7, steps)
        states.append({name: sim.get_slots(name) for name in FIELDS})
        sim.close()
    for name in FIELDS:
        assert np.isfinite(states[0][name]).all(), name
        for other in states[1:]:
            np.testing.assert_array_equal(other[name], states[0][name])
