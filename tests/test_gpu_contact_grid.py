"""The pair search's grids and the narrow phase's shortcut (GPU).

The search files the capsules in a bucket a cell or in a hash table, by FP32
or (far from the origin, where their rounding is not small against a capsule)
by FP64 corners, in cells of one or two of the largest extents as the density
suggests.  Whatever the grid, the pairs are the exhaustive search's.  The
narrow phase leaves out consecutive capsules of a rod where they cannot touch;
short elements (where its tolerance decides) and folded rods must be
evaluated, so the loads equal the oracle's there too."""
import numpy as np
import pytest

import elasticapp_b200 as eb
from elasticapp_b200 import workloads as W
from oracle_bridge import contact_spec, oracle_from_workload

pytestmark = pytest.mark.gpu

STATE = (("Position", "x"), ("Velocity", "v"), ("Director", "Q"), ("AngularVelocity", "w"))


def state_of(sim, rods):
    for name, key in STATE:
        rods.arrays[key][:] = sim.get_slots(name).reshape(-1)
    return rods


# dense grid, dense grid at FP32's limit, FP64 cells, hashed, packed (cells of
# one extent after the first step)
@pytest.mark.parametrize("box,shift", [(0.2, 0.0), (0.2, 1e3), (0.2, 3e5), (15.0, 0.0), (0.02, 0.0)])
def test_pairs_are_the_exhaustive_search(oracle_mod, box, shift):
    wl = W.contact_batch(n_rods=40, seed=17, box=box, dt=1e-9, n_elements=33)
    sim = wl.build()
    x = sim.get_slots("Position")
    x[0] += shift
    sim.set_slots("Position", x)
    rods, spec, t = oracle_from_workload(wl), contact_spec(wl), 0.0
    for _ in range(3):
        want = oracle_mod.contact_pairs(state_of(sim, rods), spec, 0.5 * wl.dt, exhaustive=True)
        t = sim.step(eb.PositionVerlet(), t, wl.dt, 1)
        assert np.array_equal(sim.contact_pairs(), want)
    sim.close()


@pytest.mark.parametrize("length", [6 * 4e-4, 6 * 3e-3])
@pytest.mark.parametrize("turn", [0.3, 1.5, 3.05, np.pi])
def test_loads_of_short_and_folded_rods(oracle_mod, length, turn):
    wl = W.contact_batch(n_rods=24, seed=18, box=4 * length, dt=1e-10, n_elements=6, length=length)
    sim = wl.build()
    x = sim.get_slots("Position")
    offs, rng = sim.slot_offsets(), np.random.default_rng(19)
    for r in range(len(wl.rods)):
        # consecutive elements turned by `turn` against one another in a random plane
        u, v = np.linalg.qr(rng.standard_normal((3, 2)))[0].T
        for i in range(6):
            d = np.cos(turn * (i % 2)) * u + np.sin(turn * (i % 2)) * v
            x[:, offs[r] + i + 1] = x[:, offs[r] + i] + d * (length / 6)
    sim.set_slots("Position", x)
    rods, spec = oracle_from_workload(wl), contact_spec(wl)
    state_of(sim, rods)
    sim.step(eb.PositionVerlet(), 0.0, wl.dt, 1)
    oracle_mod.contact_step(rods, spec, wl.dt, 1)
    for name, want in (("ContactForce", spec.capsule_force), ("ContactTorque", spec.capsule_torque)):
        want = want.reshape(3, -1)
        assert np.abs(want).max() > 0.0
        got = sim.get_slots(name)
        for r in range(len(wl.rods)):
            mine = slice(int(offs[r]), int(offs[r]) + 6)
            np.testing.assert_array_equal(got[:, mine], want[:, mine])
    sim.close()
