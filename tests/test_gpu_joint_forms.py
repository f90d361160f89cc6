"""Connections: the one-launch form (few joints a slot) and the two-launch form
(many) against the CPU restatement (GPU)."""
import numpy as np
import pytest

import elasticapp_b200 as eb
import oracle_bridge as B
from elasticapp_b200 import workloads as W

pytestmark = pytest.mark.gpu

STATE = (("Position", 0), ("Velocity", 0), ("Director", 1), ("AngularVelocity", 1))


@pytest.mark.parametrize("spokes", [1, 8, 9, 20])
def test_a_node_with_many_joints(spokes):
    rng = np.random.default_rng(31)
    n = 6

    def rod(d, m):
        return eb.StraightRod(n_elements=n, material=eb.Material(1000.0, 1e6, 1e6 / 3), radius=0.01, length=0.1,
                              origin=tuple(rng.uniform(-0.02, 0.02, 3)), direction=d, normal=m)

    rods = [rod((1, 0, 0), (0, 1, 0))] + [rod((0, 1, 0), (0, 0, 1)) for _ in range(spokes)]
    vel = [rng.normal(0, 1e-2, (3, n + 1)) for _ in rods]
    joints = [(0, 2, k + 1, 0, eb.HingeJoint(1e3, -0.1, 5.0, (0.0, 1.0, 0.0)) if k % 2 else eb.FreeJoint(2e3, -0.2))
              for k in range(spokes)]
    wl = W.Workload("star", 0, rods, clamp=[True] + [False] * spokes, damper=None, gravity=(0.0, 0.0, -9.81),
                    velocities=vel, dt=1e-5, connections=joints)
    sim = wl.build()
    sim.step(eb.PositionVerlet(), 0.0, wl.dt, 200)
    base, spread = B.oracle_spread_loads(wl, 200)
    bounds, want = B.parity_bounds(spread), B.state_slots(base)
    for name, place in STATE:
        err = B.max_rel_error_per_rod(sim.get_slots(name), want[name], wl.n_elements, place)
        assert err <= bounds[name], (name, float(err), bounds[name])
    sim.close()
