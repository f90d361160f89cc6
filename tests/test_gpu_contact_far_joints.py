"""Joints of rods with elements of kilometres, 1000 km from the origin (GPU).

The ends of consecutive capsules of a rod part by the rounding of the
coordinates; times the elements' length this passes the narrow phase's
tolerance of 1e-8 m^2 on the projections, and a few joints in a million then
touch in its arithmetic.  The loads are the oracle's there too."""
import numpy as np
import pytest

import elasticapp_b200 as eb
from elasticapp_b200 import workloads as W
from oracle_bridge import contact_spec, oracle_from_workload

pytestmark = pytest.mark.gpu

# nodes of two elements that touch so
JOINTS = (
    "-0x1.d031696d24653p+17 0x1.f7a7717729082p+18 -0x1.40ce99204fef8p+19 -0x1.cb6d39ce15a3bp+17 0x1.efee24f3745f8p+18 -0x1.40dc84cd3ff8dp+19 -0x1.c5d356558aff4p+17 0x1.e7118df5a37d4p+18 -0x1.40e31efa1e179p+19",
    "-0x1.1ad68353de649p+19 -0x1.cd5fdd7597ca4p+19 0x1.197d4cf6a56e1p+18 -0x1.1b4edf5b625dep+19 -0x1.cd4090c0b1e66p+19 0x1.10969949026dep+18 -0x1.1bd97bb6c397p+19 -0x1.cd1a662a81d1fp+19 0x1.072b1a0736456p+18",
    "0x1.20a88a0021446p+18 0x1.7b87fb732f56p+19 -0x1.7ef2f5e0e0ae7p+18 0x1.229a3b83e5a31p+18 0x1.7c0a9fccc7c3dp+19 -0x1.79731a8ca3121p+18 0x1.2587583c2b1ebp+18 0x1.7cc826bb55f9ep+19 -0x1.713e8d73f4ef6p+18",
    "-0x1.94b512947af4p+19 -0x1.556be2c82535p+19 -0x1.7a1976d8c9f2p+18 -0x1.93a635e395a31p+19 -0x1.59a222e099f0ep+19 -0x1.7ae68fd3b40d1p+18 -0x1.927957e5cea63p+19 -0x1.5e2525f6009d1p+19 -0x1.7bc6a3a35c25cp+18",
    "-0x1.e1b38294c2631p+19 0x1.33018ed5ef0d1p+19 -0x1.3170cca25a336p+19 -0x1.de057d37aa41p+19 0x1.3251e110cbbbdp+19 -0x1.326263975f044p+19 -0x1.d98b48cea153p+19 0x1.3176e6a1fe526p+19 -0x1.338f5d589e675p+19",
)


def test_loads_of_long_elements_far_out(oracle_mod):
    wl = W.contact_batch(n_rods=len(JOINTS), seed=18, box=1.0, dt=1e-10, n_elements=2, length=18000.0)
    wl.velocities = [np.zeros((3, 3)) for _ in JOINTS]
    wl.planes = []
    sim = wl.build()
    x = sim.get_slots("Position")
    for o, joint in zip(sim.slot_offsets(), JOINTS):
        x[:, o:o + 3] = np.array([float.fromhex(t) for t in joint.split()]).reshape(3, 3).T
    sim.set_slots("Position", x)
    rods, spec = oracle_from_workload(wl), contact_spec(wl)
    for name, key in (("Position", "x"), ("Velocity", "v"), ("Director", "Q"), ("AngularVelocity", "w")):
        rods.arrays[key][:] = sim.get_slots(name).reshape(-1)
    sim.step(eb.PositionVerlet(), 0.0, wl.dt, 1)
    oracle_mod.contact_step(rods, spec, wl.dt, 1)
    for name, want in (("ContactForce", spec.capsule_force), ("ContactTorque", spec.capsule_torque)):
        want = want.reshape(3, -1)
        got = sim.get_slots(name)
        for o in sim.slot_offsets()[:-1]:
            mine = slice(int(o), int(o) + 2)
            assert np.abs(want[:, mine]).max() > 0.0
            np.testing.assert_array_equal(got[:, mine], want[:, mine])
    sim.close()
