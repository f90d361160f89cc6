"""Served rods: the initial data written on the device and the results written
to the host arena are those of a simulator holding the same rods (GPU).

Both run the resident FP64 kernel, whose arithmetic does not depend on what
else a CTA holds, so the states are equal bit for bit."""
import numpy as np
import pytest

import elasticapp_b200 as eb
from elasticapp_b200.server import Server

pytestmark = pytest.mark.gpu

FIELDS = ("Position", "Velocity", "Director", "AngularVelocity")


def random_rods(lengths, rng):
    rods = []
    for n in lengths:
        d = rng.standard_normal(3)
        c = rng.standard_normal(3)
        for _ in range(2):
            c = c - (c @ d) / (d @ d) * d
        rods.append(eb.StraightRod(int(n), eb.Material(rng.uniform(800, 1200), 1e6, 3e5), rng.uniform(0.01, 0.03),
                                   rng.uniform(0.5, 1.5), tuple(rng.uniform(-1, 1, 3)), tuple(d), tuple(c), 0.3, 0.2))
    return rods


@pytest.mark.parametrize("model", [eb.CosseratRodWithoutDamping, eb.CosseratRod])
@pytest.mark.parametrize("moving", [False, True])
@pytest.mark.parametrize("requests", [[[2, 3], [519]], [[255, 256, 257, 2], [700, 5], [1039]]])
def test_results_equal_a_simulator(model, moving, requests):
    rng = np.random.default_rng(61)
    srv, cases = Server(precision="fp64", hbm_budget_bytes=2e8, steps_per_launch=16), []
    for lengths in requests:
        rods = random_rods(lengths, rng)
        vel = [rng.normal(0, 1e-2, (3, n + 1)) for n in lengths] if moving else None
        rid = srv.submit(rods, dt=1e-6, n_steps=40, gravity=(0.0, 0.3, -9.81), clamp=True, damper=(0.1, 0.2),
                         velocities=vel, model=model)
        cases.append((rid, rods, vel))
    srv.run_until_idle()
    for rid, rods, vel in cases:
        sim = eb.Simulator(step_mode="bucketed" if max(r.n_elements for r in rods) > 519 else "resident")
        refs = sim.emplace_back_many(model, rods)
        sim.add_environment(eb.GravityField((0.0, 0.3, -9.81)))
        for k, ref in enumerate(refs):
            if vel is not None:
                ref.set("Velocity", vel[k])
            sim.constrain(ref).at(0).using(eb.Clamp())
            sim.constrain(ref).using(eb.AnalyticalLinearDamper(0.1, 0.2))
        sim.finalize()
        sim.step(eb.PositionVerlet(), 0.0, 1e-6, 40)
        for k, ref in enumerate(refs):
            for name in FIELDS:
                assert np.array_equal(srv.result(rid, k, name), ref.get(name)), (name, k)
        sim.close()
    srv.close()
