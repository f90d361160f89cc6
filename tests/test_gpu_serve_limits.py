"""The server at its limits (GPU): requests whose initial data need several
stages."""
import numpy as np
import pytest

import elasticapp_b200 as eb
from elasticapp_b200.server import Server

pytestmark = pytest.mark.gpu

FIELDS = ("Position", "Velocity", "Director", "AngularVelocity")


def rod(n, k=0):
    return eb.StraightRod(n, eb.Material(1000.0, 1e6, 3e5), 0.01, 1.0, origin=(0.0, 1e-3 * k, 0.0))


def test_admission_in_several_stages():
    """5500 rods of 1040 slots with velocities, 137 MB of initial data."""
    rng = np.random.default_rng(81)
    n_rods, n = 5500, 1039
    rods = [rod(n, k) for k in range(n_rods)]
    vel = list(rng.normal(0.0, 1e-2, (n_rods, 3, n + 1)))
    args = dict(dt=1e-7, n_steps=3, gravity=(0.0, 0.0, -9.81), clamp=True, damper=(0.1, 0.1))
    srv = Server(precision="fp64", hbm_budget_bytes=5e9)
    small = srv.submit([rod(20)], **args)
    rid = srv.submit(rods, velocities=vel, **args)
    assert {c["request_id"] for c in srv.run_until_idle()} == {small, rid}
    for k in (0, 1, 2600, 2800, n_rods - 1):
        alone = srv.submit([rods[k]], velocities=[vel[k]], **args)
        srv.run_until_idle()
        for name in FIELDS:
            assert np.array_equal(srv.result(rid, k, name), srv.result(alone, 0, name)), (k, name)
    srv.close()
