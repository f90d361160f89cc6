"""A node of infinite mass keeps its velocity under every plan (GPU): its
acceleration is the load divided by infinity, zero."""
import numpy as np
import pytest

import elasticapp_b200 as eb

pytestmark = pytest.mark.gpu

MODES = [dict(step_mode="streaming"), dict(step_mode="resident", resident_config=3),
         dict(step_mode="resident", resident_config=2)]


# rods of fewer slots than a CTA's threads, and (520 slots on 256 threads) of more
@pytest.mark.parametrize("lengths", [(12, 5), (300,)])
@pytest.mark.parametrize("mode", MODES, ids=["streaming", "264", "520"])
@pytest.mark.parametrize("mass", [np.inf, 1e200])
def test_infinite_mass_keeps_its_velocity(lengths, mode, mass):
    if mode.get("resident_config") == 3 and max(lengths) > 263:
        pytest.skip("longer than the configuration's CTA")
    rods = [eb.StraightRod(n, eb.Material(1000.0, 1e6, 3e5), 0.01, 1.0, origin=(0.0, 0.3 * k, 0.0))
            for k, n in enumerate(lengths)]
    sim = eb.Simulator(**mode)
    refs = sim.emplace_back_many(eb.CosseratRodWithoutDamping, rods)
    sim.finalize()
    rng = np.random.default_rng(71)
    v = rng.normal(0.0, 1e-2, (3, sim.n_slots()))
    sim.set_slots("Velocity", v)
    m = sim.get_slots("Mass")
    held = [int(o) + n // 2 for o, n in zip(sim.slot_offsets(), lengths)]
    m[:, held] = mass
    sim.set_slots("Mass", m)
    sim.step(eb.PositionVerlet(), 0.0, 1e-6, 50)
    for ref in refs:
        for name in ("Position", "Velocity", "Director", "AngularVelocity"):
            assert np.isfinite(ref.get(name)).all(), name
    np.testing.assert_array_equal(sim.get_slots("Velocity")[:, held], v[:, held])
    sim.close()
