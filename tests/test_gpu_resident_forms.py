"""Resident FP64 kernel: its forms agree bit for bit (GPU).

A CTA of at most as many slots as threads keeps a slot in its thread's
registers; a longer one steps several slots a thread from shared memory.
Configurations 1 to 4 (520 slots on 512 or 256 threads, 264 on 256, 320 on
320) put the same rods into either form, so their states must be equal; a
run cut into several calls, and directors turned past the small-angle and
below the guarded range, go through the same comparison."""
import numpy as np
import pytest

import elasticapp_b200 as eb
from elasticapp_b200 import workloads as W

pytestmark = pytest.mark.gpu

FIELDS = ("Position", "Velocity", "Director", "AngularVelocity")


def run(wl, config, stepper, omega, calls):
    sim = wl.build(resident_config=config, step_mode="resident", stepper=stepper)
    rng = np.random.default_rng(3)
    sim.set_slots("AngularVelocity", rng.normal(0.0, 1.0, (3, sim.n_slots())) * omega)
    t = 0.0
    for k in calls:
        t = sim.step(stepper(), t, wl.dt, k)
    out = {name: sim.get_slots(name) for name in FIELDS}
    sim.close()
    return out


@pytest.mark.parametrize("stepper", [eb.PositionVerlet, eb.VelocityVerlet, eb.PEFRL])
@pytest.mark.parametrize("lengths", [[2, 3, 263, 255, 256, 7], [31, 32, 33, 64, 200]])
@pytest.mark.parametrize("omega", [0.0, 1e-9, 3.0, 3e5])
def test_configurations_agree_bit_for_bit(stepper, lengths, omega):
    wl = W.uneven_batch(n_rods=len(lengths), seed=11, n_range=(2, 2))
    rng = np.random.default_rng(12)
    for rod, n in zip(wl.rods, lengths):
        rod.n_elements = n
    wl.velocities = [rng.normal(0.0, 1e-3, size=(3, n + 1)) for n in lengths]
    wl.dt = 1e-7
    want = run(wl, 1, stepper, omega, (9,))
    for config, calls in ((1, (4, 5)), (2, (9,)), (3, (9,)), (4, (2, 7))):
        got = run(wl, config, stepper, omega, calls)
        for name in FIELDS:
            assert np.array_equal(got[name], want[name], equal_nan=True), (name, config)
