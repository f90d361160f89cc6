"""The server at its limits (GPU): device memory within the budget, requests
whose initial data need several stages, results that cannot be delivered or
wait for room."""
import numpy as np
import pytest

import elasticapp_b200 as eb
from elasticapp_b200.server import Server

pytestmark = pytest.mark.gpu

FIELDS = ("Position", "Velocity", "Director", "AngularVelocity")


def rod(n, k=0):
    return eb.StraightRod(n, eb.Material(1000.0, 1e6, 3e5), 0.01, 1.0, origin=(0.0, 1e-3 * k, 0.0))


def test_device_memory_within_the_budget():
    import torch

    Server(hbm_budget_bytes=2e8).close()  # the context and the module
    before, _ = torch.cuda.mem_get_info(0)
    srv = Server(hbm_budget_bytes=2e8)
    after, _ = torch.cuda.mem_get_info(0)
    srv.close()
    # 14 allocations, each rounded up to a granule of 2 MiB
    assert before - after <= 2e8 + 28 * 2 ** 20


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


def test_undeliverable_result_stops_no_other():
    """A result larger than the host arena (1 GiB) fails every tick; the
    requests that finish with it, or later, are delivered."""
    args = dict(dt=1e-7, n_steps=2, gravity=(0.0, 0.0, -9.81), clamp=True)
    srv = Server(precision="fp64", hbm_budget_bytes=5e9, steps_per_launch=2)
    first = srv.submit([rod(30)], **args)
    big = srv.submit([rod(1039, k) for k in range(7500)], **args)
    same, later = srv.submit([rod(20)], **args), srv.submit([rod(25)], **dict(args, n_steps=9))
    done = set()
    for _ in range(50):
        with pytest.raises(Exception, match="arena"):
            srv.tick()
        done |= {c["request_id"] for c in srv.poll()}
        if done == {first, same, later}:
            break
    assert done == {first, same, later}
    assert srv.request_status(big)["state"] == "active"
    assert srv.stats()["bins_used"] == 15000
    ref = Server(precision="fp64", hbm_budget_bytes=2e8, steps_per_launch=2)
    for rid, n, steps in ((first, 30, 2), (same, 20, 2), (later, 25, 9)):
        alone = ref.submit([rod(n)], **dict(args, n_steps=steps))
        ref.run_until_idle()
        for name in FIELDS:
            assert np.array_equal(srv.result(rid, 0, name), ref.result(alone, 0, name)), (n, name)
    ref.close()
    srv.close()


def test_results_wait_for_room_in_the_arena():
    """Three results of 494 MB that finish together pass through the arena of 1 GiB."""
    args = dict(dt=1e-7, n_steps=3, gravity=(0.0, 0.0, -9.81), clamp=True)
    srv = Server(precision="fp64", hbm_budget_bytes=8e9, steps_per_launch=2)
    ids = [srv.submit([rod(1039, 10000 * i + k) for k in range(3300)], **args) for i in range(3)]
    assert {c["request_id"] for c in srv.run_until_idle()} == set(ids)
    for i, rid in enumerate(ids):
        for k in (0, 3299):
            alone = srv.submit([rod(1039, 10000 * i + k)], **args)
            srv.run_until_idle()
            for name in FIELDS:
                assert np.array_equal(srv.result(rid, k, name), srv.result(alone, 0, name)), (i, k, name)
    srv.close()


def test_a_million_rods():
    """Specifications and result lists of a million rods, in several stages each."""
    args, n_rods = dict(dt=1e-7, n_steps=3, gravity=(0.0, 0.0, -9.81), clamp=True), 1_000_000
    srv = Server(precision="fp64", hbm_budget_bytes=8e9, steps_per_launch=2)
    kinds = [rod(2, k) for k in range(7)]
    rid = srv.submit([kinds[k % 7] for k in range(n_rods)], **args)
    srv.run_until_idle()
    for kind in range(7):
        alone = srv.submit([kinds[kind]], **args)
        srv.run_until_idle()
        for k in [kind, *range(kind + 7 * 20_000, n_rods, 7 * 20_000), kind + (n_rods - 1 - kind) // 7 * 7]:
            for name in FIELDS:
                assert np.array_equal(srv.result(rid, k, name), srv.result(alone, 0, name)), (k, name)
    srv.close()
