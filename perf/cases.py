"""Timed cases of the rod framework: the calls that its users' programs make,
over the sizes that the workloads, tests and benchmark of this repository use.

Four kinds of program:

* ``rods``    - a batch of independent rods stepped through ``Simulator.step``
  and read back with ``Simulator.step_host_state`` (the loop of a case study:
  set up, run, communicate).  From the single cantilever of 100 elements to
  8,192 rods of 32 to 512 elements; FP64 and mixed precision; rods with and
  without explicit damping; straight rods and rods with rest curvature and an
  end torque; the three steppers; one long call or many calls of one step;
  the state set from the host at every pass or kept on the device.
* ``contact`` - free rods in a box whose elements collide with one another
  and with the walls (the collision system).
* ``chain``   - rods joined end to end by hinges (connections).
* ``serve``   - a burst of requests through the continuous-batching server.

A pass goes on from the state the last pass left, as a simulation does; time
steps are below the stability bounds of the stiffest rod, so a state stays
finite over any number of passes.
"""
import math

import numpy as np
import torch

import elasticapp_b200 as eb
from elasticapp_b200.server import Server

STATE = ("Position", "Velocity", "Director", "AngularVelocity")
WIDTH = {"Position": 3, "Velocity": 3, "Director": 9, "AngularVelocity": 3}
STEPPERS = {"position_verlet": eb.PositionVerlet, "pefrl": eb.PEFRL, "velocity_verlet": eb.VelocityVerlet}
EVALUATIONS = {"position_verlet": 1, "pefrl": 4, "velocity_verlet": 2}
DENSITY = 1000.0
DAMPER = (0.1, 0.1)
EXPLICIT_DAMPING = 0.5
CLAMP_GRAVITY = (0.0, 0.0, -9.81)


def _rods(name, rods, lo, hi, calls, steps, stepper="position_verlet", precision="fp64", rod="plain",
          rest="straight", host=False):
    case = {"kind": "rods", "rods": rods, "lo": lo, "hi": hi, "calls": calls, "steps": steps, "stepper": stepper,
            "precision": precision, "rod": rod, "rest": rest, "host": host}
    return dict(case, name=name) if name else case


def listed():
    return [
        # one cantilever, a callback after every step: the smallest calls, bound by launch latency
        _rods("cantilever_step_calls", 1, 100, 100, calls=32, steps=1),
        # the same cantilever run for a long time in one call (the reference's dynamic cantilever example)
        _rods("cantilever_run", 1, 100, 100, calls=1, steps=2000),
        # a study of a few dozen rods of odd sizes: fills a small part of the chip
        _rods("family_run", 61, 37, 203, calls=1, steps=400),
        # the headline batch shape, many steps between read-backs
        _rods("uneven_run", 8192, 32, 512, calls=1, steps=128),
        # the same shape driven one step a call, as by a program with its own rule between steps
        _rods("uneven_step_calls", 4096, 32, 512, calls=64, steps=1),
        # a host-driven loop: state in from host memory and out again every cycle
        _rods("host_cycle", 4096, 32, 512, calls=1, steps=100, host=True),
        # mixed precision, rest curvature and end torque
        _rods("mixed_run", 8192, 64, 256, calls=1, steps=128, precision="mixed", rest="curved"),
        # the fourth-order stepper
        _rods("pefrl_run", 2048, 32, 512, calls=1, steps=32, stepper="pefrl"),
        # long explicitly damped rods, each over two CTAs
        _rods("damped_long_run", 512, 520, 1039, calls=1, steps=64, rod="damped"),
        # colliding rods: half a million capsules, and the walls of the box
        {"name": "contact_run", "kind": "contact", "rods": 8192, "elements": 64, "steps": 8},
        # joints between rods
        {"name": "hinge_chain", "kind": "chain", "links": 32, "elements": 10, "steps": 100},
        # a burst of requests of rods of 32 to 1024 elements through the server
        {"name": "serve_burst", "kind": "serve", "requests": 24, "rods": 4, "lo": 32, "hi": 1024, "steps": 512},
    ]


def _between(rng, lo, hi):
    """An integer in [lo, hi], spread over the logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(("rods", "rods", "rods", "rods", "calls", "mixed", "long", "contact", "chain", "serve"))
    if kind == "contact":
        return {"kind": "contact", "rods": _between(rng, 96, 8192), "elements": rng.randint(24, 64),
                "steps": rng.randint(1, 8)}
    if kind == "chain":
        return {"kind": "chain", "links": _between(rng, 2, 64), "elements": rng.randint(6, 40),
                "steps": _between(rng, 10, 100)}
    if kind == "serve":
        return {"kind": "serve", "requests": _between(rng, 4, 24), "rods": rng.randint(1, 4), "lo": 32,
                "hi": rng.randint(200, 1024), "steps": _between(rng, 64, 512)}
    if kind == "calls":
        return _rods(None, _between(rng, 1, 2048), rng.randint(12, 64), rng.randint(65, 512),
                     calls=rng.randint(8, 64), steps=1, rod=rng.choice(("plain", "damped")))
    if kind == "long":
        return _rods(None, _between(rng, 8, 512), rng.randint(300, 600), rng.randint(601, 1039), calls=1,
                     steps=_between(rng, 16, 64), precision=rng.choice(("fp64", "mixed")),
                     rod=rng.choice(("plain", "damped")))
    if kind == "mixed":
        return _rods(None, _between(rng, 16, 8192), rng.randint(33, 100), rng.randint(101, 256), calls=1,
                     steps=_between(rng, 16, 128), precision="mixed", rest=rng.choice(("straight", "curved")))
    return _rods(None, _between(rng, 1, 4096), rng.randint(8, 100), rng.randint(101, 512), calls=1,
                 steps=_between(rng, 16, 128), stepper=rng.choice(("position_verlet", "position_verlet", "pefrl",
                                                                  "velocity_verlet")),
                 rod=rng.choice(("plain", "plain", "damped")), rest=rng.choice(("straight", "curved")),
                 host=rng.random() < 0.3)


# ---- inputs ------------------------------------------------------------------

def _unit(v):
    return v / np.linalg.norm(v, axis=1, keepdims=True)


def _frames(rng, count):
    """Random directions and normals orthogonal to them."""
    d = _unit(rng.standard_normal((count, 3)))
    c = rng.standard_normal((count, 3))
    for _ in range(2):
        c = _unit(c - np.sum(c * d, axis=1, keepdims=True) * d)
    return d, c


def _time_step(length, n, radius, E):
    """Below the axial and the bending bound of the stiffest rod."""
    ell, c = length / n, np.sqrt(E / DENSITY)
    return float(min(np.min(0.1 * ell / c), np.min(0.3 * ell * ell / (radius * c))))


def _describe(case, seed):
    """The program's inputs: per-rod parameters, the state's velocities and the modules in use."""
    rng = np.random.Generator(np.random.PCG64(seed))
    kind = case["kind"]
    w = {"rest_curvature": None, "torque": None, "explicit": 0.0, "planes": [], "contact": None, "joints": [],
         "damper": None, "gravity": CLAMP_GRAVITY}
    if kind == "contact":
        R, n = case["rods"], case["elements"]
        length, radius = 0.2, 0.0007
        side = (R / 8192.0) ** (1.0 / 3.0)  # the density of 8,192 rods in a unit cube
        w["n"] = np.full(R, n)
        w["L"], w["r"] = np.full(R, length), np.full(R, radius)
        w["E"] = np.full(R, 1e6)
        w["d"], w["normal"] = _frames(rng, R)
        centres = rng.uniform(0.0, side, (R, 3))
        w["origin"] = centres - 0.5 * length * w["d"]
        w["clamp"] = np.zeros(R, bool)
        w["contact"] = eb.ContactMaterial(stiffness=20.0, normal_damping=1e-4, tangential_damping=1e-4,
                                          static_friction=0.15, dynamic_friction=0.15)
        h = 0.5 * side
        w["planes"] = [((0.0, h, h), (1.0, 0.0, 0.0)), ((side, h, h), (-1.0, 0.0, 0.0)),
                       ((h, 0.0, h), (0.0, 1.0, 0.0)), ((h, side, h), (0.0, -1.0, 0.0)),
                       ((h, h, 0.0), (0.0, 0.0, 1.0)), ((h, h, side), (0.0, 0.0, -1.0))]
        spread, w["dt"] = 0.05, 1e-6
    elif kind == "chain":
        # the hinge-joint example's rods end to end along z
        R, n = case["links"], case["elements"]
        w["n"] = np.full(R, n)
        w["L"], w["r"], w["E"] = np.full(R, 0.2), np.full(R, 0.007), np.full(R, 3e7)
        w["d"] = np.tile([0.0, 0.0, 1.0], (R, 1))
        w["normal"] = np.tile([0.0, 1.0, 0.0], (R, 1))
        w["origin"] = np.stack([np.zeros(R), np.zeros(R), 0.2 * np.arange(R)], axis=1)
        w["clamp"] = np.arange(R) == 0
        w["explicit"], w["gravity"] = 0.015, (0.0, -9.81, 0.0)
        w["joints"] = [(k, n - 1, k + 1, 0, 1e5, 5e3, (1.0, 0.0, 0.0)) for k in range(R - 1)]
        spread = 1e-3
        w["dt"] = _time_step(w["L"], w["n"], w["r"], w["E"])
    else:
        R = case["rods"] * case.get("requests", 1)
        # the rods' sizes are the case's, whatever the seed
        sizes = np.random.Generator(np.random.PCG64([R, case["lo"], case["hi"]]))
        w["n"] = sizes.integers(case["lo"], case["hi"] + 1, R)
        if R == 1 and case["lo"] == case["hi"]:
            # the cantilever of the dynamic cantilever example
            w["L"], w["r"], w["E"] = np.ones(1), np.full(1, 0.025), np.full(1, 1e6)
            w["d"], w["normal"] = np.array([[1.0, 0.0, 0.0]]), np.array([[0.0, 1.0, 0.0]])
            w["origin"] = np.zeros((1, 3))
        else:
            w["L"] = rng.uniform(0.5, 2.0, R)
            w["r"] = rng.uniform(0.005, 0.05, R)
            w["E"] = 10.0 ** rng.uniform(5.0, 7.0, R)
            w["d"], w["normal"] = _frames(rng, R)
            w["origin"] = rng.uniform(-1.0, 1.0, (R, 3))
        w["clamp"], w["damper"] = np.ones(R, bool), DAMPER
        if case.get("rod") == "damped":
            w["explicit"] = EXPLICIT_DAMPING
        if case.get("rest") == "curved":
            w["rest_curvature"] = rng.uniform(0.0, 10.0, (R, 1)) * _unit(rng.standard_normal((R, 3)))
            w["torque"] = 1e-3 * w["d"]
        spread = 1e-3
        w["dt"] = _time_step(w["L"], w["n"], w["r"], w["E"])
    w["slots"] = int(np.sum(w["n"] + 1))
    w["velocity"] = rng.normal(0.0, spread, (3, w["slots"]))
    return w


def _modulus(case, w):
    """Shear modulus: two thirds of E for the hinge example's material, E / 3 otherwise."""
    return w["E"] * (2.0 / 3.0 if case["kind"] == "chain" else 1.0 / 3.0)


def _density(case):
    return 1750.0 if case["kind"] == "chain" else DENSITY


def _initializers(case, w):
    G, rho = _modulus(case, w), _density(case)
    return [eb.StraightRod(n_elements=int(w["n"][k]), material=eb.Material(rho, float(w["E"][k]), float(G[k])),
                           radius=float(w["r"][k]), length=float(w["L"][k]), origin=w["origin"][k],
                           direction=w["d"][k], normal=w["normal"][k], force_damping_rate=w["explicit"],
                           torque_damping_rate=w["explicit"]) for k in range(len(w["n"]))]


def _rod_of_slot(w):
    return np.repeat(np.arange(len(w["n"])), w["n"] + 1)


def _first_slots(w):
    return np.concatenate([[0], np.cumsum(w["n"] + 1)])


def prepare(case, seed):
    w = _describe(case, seed)
    inits = _initializers(case, w)
    if case["kind"] == "serve":
        server = Server(precision="mixed", hbm_budget_bytes=2e9)
        k, first, requests = case["rods"], _first_slots(w), []
        for q in range(case["requests"]):
            mine = range(q * k, (q + 1) * k)
            requests.append(([inits[r] for r in mine], [w["velocity"][:, first[r]:first[r + 1]] for r in mine]))
        return {"kind": "serve", "server": server, "requests": requests, "dt": w["dt"], "steps": case["steps"]}
    sim = eb.Simulator(precision=case.get("precision", "fp64"), stepper=STEPPERS[case.get("stepper", "position_verlet")])
    damped = case["kind"] == "chain" or case.get("rod") == "damped"
    refs = sim.emplace_back_many(eb.CosseratRod if damped else eb.CosseratRodWithoutDamping, inits)
    sim.add_environment(eb.GravityField(w["gravity"]))
    for k, ref in enumerate(refs):
        if w["clamp"][k]:
            sim.constrain(ref).at(0).using(eb.Clamp())
        if w["damper"] is not None:
            sim.constrain(ref).using(eb.AnalyticalLinearDamper(*w["damper"]))
        if w["torque"] is not None:
            sim.force(ref).using(eb.EndTorque(w["torque"][k]))
    if w["contact"] is not None:
        sim.add_environment(eb.CollisionSystem())
        material = sim.create_material(w["contact"])
        for ref in refs:
            sim.add_contact(ref, material)
        for point, normal in w["planes"]:
            sim.emplace_plane(point, normal, material)
    for ra, ia, rb, ib, k, k_rot, normal in w["joints"]:
        sim.connect(refs[ra], ia).to(refs[rb], ib).using(eb.HingeJoint(k, 0.0, k_rot, normal))
    sim.finalize()
    sim.set_slots("Velocity", w["velocity"])
    if w["rest_curvature"] is not None:
        kap = w["rest_curvature"][_rod_of_slot(w)].T
        kap = np.where(_masks(w)["voronoi"], kap, 0.0)
        sim.set_slots("ReferenceCurvature", kap)

    def pinned(name):
        return torch.empty((WIDTH[name], w["slots"]), dtype=torch.float64,
                           pin_memory=torch.cuda.is_available()).numpy()

    # the host's arrays of the state, pinned as a program that exchanges them would have them
    out = {name: pinned(name) for name in STATE}
    inputs = None
    if case.get("host"):
        inputs = {name: pinned(name) for name in STATE}
        for name in STATE:
            sim.get_slots(name, out=inputs[name])
    return {"kind": case["kind"], "sim": sim, "dt": w["dt"], "steps": case["steps"], "calls": case.get("calls", 1),
            "inputs": inputs, "out": out, "stepper": STEPPERS[case.get("stepper", "position_verlet")](), "time": 0.0}


def run(state):
    if state["kind"] == "serve":
        return _serve(state)
    sim, stepper, dt, t = state["sim"], state["stepper"], state["dt"], state["time"]
    for _ in range(state["calls"] - 1):
        t = sim.step(stepper, t, dt, state["steps"])
    state["time"] = sim.step_host_state(stepper, t, dt, state["steps"], inputs=state["inputs"], outputs=state["out"])
    if state["kind"] == "contact":
        return dict(state["out"], ContactForce=sim.get_slots("ContactForce"))
    return dict(state["out"])


def _serve(state):
    server = state["server"]
    ids = [server.submit(rods, dt=state["dt"], n_steps=state["steps"], gravity=CLAMP_GRAVITY, clamp=True,
                         damper=DAMPER, velocities=velocities) for rods, velocities in state["requests"]]
    while server.tick():
        server.poll()
    server.poll()
    out = {name: np.concatenate([server.result(i, k, name).reshape(WIDTH[name], -1)
                                 for i, (rods, _) in zip(ids, state["requests"]) for k in range(len(rods))], axis=1)
           for name in STATE}
    for i in ids:
        server.release(i)
    return out


def work(case):
    """One pass: per call every rod's state read and written once and its parameters read once (18 state values
    and 22 parameters a slot), and about 500 operations an element and force evaluation."""
    if case["kind"] in ("contact", "chain"):
        rods, mean, calls = case.get("rods", case.get("links")), case["elements"], 1
    else:
        rods, mean, calls = case["rods"] * case.get("requests", 1), 0.5 * (case["lo"] + case["hi"]), case.get("calls", 1)
    evaluations = EVALUATIONS[case.get("stepper", "position_verlet")]
    slots = rods * (mean + 1)
    return {"bytes": 8.0 * slots * (36 + 22) * calls, "flops": 500.0 * rods * mean * calls * case["steps"] * evaluations}


# ---- the same in plain 64-bit torch --------------------------------------------

def _masks(w):
    first = _first_slots(w)
    j = np.arange(w["slots"]) - np.repeat(first[:-1], w["n"] + 1)
    n = np.repeat(w["n"], w["n"] + 1)
    return {"j": j, "element": j < n, "voronoi": j < n - 1, "first": j == 0, "last_element": j == n - 1}


def _cross(a, b):
    return torch.stack([a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]])


def _dot(a, b):
    return (a * b).sum(0)


def _next(a):
    """Entry of the slot to the right (the last slot's is its own and never used)."""
    return torch.cat([a[..., 1:], a[..., -1:]], dim=-1)


def _before(a):
    """Entry of the slot to the left, zero for the first slot."""
    return torch.cat([torch.zeros_like(a[..., :1]), a[..., :-1]], dim=-1)


def _rotate(Q, u):
    """exp(-[u]x) Q with the axis u / (|u| + 1e-14)."""
    theta = u.square().sum(0).sqrt()
    c, s = torch.cos(theta), torch.sin(theta)
    one_minus_c = 2.0 * torch.sin(0.5 * theta).square()
    u = u / (theta + 1e-14)
    along = (u[:, None] * Q).sum(0)
    turn = torch.stack([Q[1] * u[2] - Q[2] * u[1], Q[2] * u[0] - Q[0] * u[2], Q[0] * u[1] - Q[1] * u[0]])
    return c * Q + one_minus_c * u[:, None] * along[None] + s * turn


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


class _Plain:
    """The rods' step in 64-bit torch operations over all slots (a slot holds a node, an element and a Voronoi
    point of its rod)."""

    def __init__(self, case, w):
        dev = _device()
        put = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=dev)  # noqa: E731
        m = _masks(w)
        self.w, self.dt = w, w["dt"]
        rod = _rod_of_slot(w)
        self.E, self.V = (torch.as_tensor(m[k], device=dev) for k in ("element", "voronoi"))
        self.first, self.last = (torch.as_tensor(m[k], device=dev) for k in ("first", "last_element"))
        self.not_first = (~self.first).to(torch.float64)
        d, normal = w["d"], w["normal"]
        d = d / np.linalg.norm(d, axis=1, keepdims=True)
        normal = normal / np.linalg.norm(normal, axis=1, keepdims=True)
        step = ((w["origin"] + w["L"][:, None] * d) - w["origin"]) / w["n"][:, None]
        self.x = put((w["origin"][rod] + m["j"][:, None] * step[rod]).T)
        third = np.cross(normal, np.cross(d, normal))
        second = np.cross(third, normal)
        third, second = _unit(third), _unit(second)
        self.Q = torch.where(self.E, put(np.stack([normal, second, third], 1)[rod].transpose(1, 2, 0)), 0.0)
        self.v, self.omega = put(w["velocity"]), torch.zeros_like(self.x)
        dx = _next(self.x) - self.x
        one = torch.ones((), dtype=torch.float64, device=dev)
        self.l0 = torch.where(self.E, dx.square().sum(0).sqrt(), one)
        self.D0 = torch.where(self.V, 0.5 * (self.l0 + _next(self.l0)), one)
        radius, young = put(w["r"][rod]), put(w["E"][rod])
        shear, rho = put(_modulus(case, w)[rod]), _density(case)
        area = math.pi * radius.square()
        I1 = area.square() / (4.0 * math.pi)
        I = torch.stack([I1, I1, 2.0 * I1])
        self.volume = area * self.l0
        self.S = torch.stack([shear, shear, young]) * area * torch.tensor(
            [[13.5 / 14.0], [13.5 / 14.0], [1.0]], dtype=torch.float64, device=dev)
        self.B = torch.stack([young, young, shear]) * I
        self.J = I * rho * self.l0
        half = torch.where(self.E, 0.5 * rho * self.volume, 0.0)
        self.mass = half + _before(half) * self.not_first
        self.kap0 = torch.zeros_like(self.x)
        if w["rest_curvature"] is not None:
            self.kap0 = torch.where(self.V, put(w["rest_curvature"][rod].T), 0.0)
        self.torque = None
        if w["torque"] is not None:
            self.torque = torch.where(self.last, put(w["torque"][rod].T), 0.0)
        self.clamped = self.first & torch.as_tensor(w["clamp"][rod], device=dev)
        self.x_clamp, self.Q_clamp = self.x.clone(), self.Q.clone()
        self.gravity = put(w["gravity"])[:, None]
        em = 0.5 * (self.mass + _next(self.mass)) + 0.5 * self.mass * self.first + 0.5 * _next(self.mass) * self.last
        self.element_mass = em
        self.contact = _Contact(self, dev) if w["contact"] is not None else None
        self.joints = w["joints"]
        if self.joints:
            at = _first_slots(w)
            ja = np.array([[at[ra] + ia, at[rb] + ib] for ra, ia, rb, ib, *_ in self.joints])
            self.ja, self.jb = (torch.as_tensor(ja[:, k], device=dev) for k in (0, 1))
            self.jk, self.jrot = self.joints[0][4], self.joints[0][5]
            self.jn = put(self.joints[0][6])[:, None]

    def drift(self, c):
        self.x = self.x + c * self.v
        self.Q = torch.where(self.E, _rotate(self.Q, c * self.omega), self.Q)

    def clamp(self):
        self.x = torch.where(self.clamped, self.x_clamp, self.x)
        self.Q = torch.where(self.clamped, self.Q_clamp, self.Q)

    def kick(self, dt, damper_dt, x_rate):
        E, V, x, Q, w = self.E, self.V, self.x, self.Q, self.omega
        zero = torch.zeros((), dtype=torch.float64, device=x.device)
        dx = _next(x) - x
        l = torch.where(E, dx.square().sum(0).sqrt(), 1.0)
        t, e = dx / l, l / self.l0
        qt = (Q * t[None]).sum(1)
        strain = qt * e
        strain = torch.stack([strain[0], strain[1], strain[2] - 1.0])
        stress = torch.where(E, self.S * strain, zero)
        force = torch.where(E, (Q * stress[:, None]).sum(0) / e, zero)
        F = force - _before(force) * self.not_first
        if self.w["explicit"]:
            F = F - self.mass * self.w["explicit"] * self.v
        F = F + self.gravity * self.mass
        Jwe = self.J * w / e
        rate = _dot(t, _next(self.v) - self.v) / l
        T = _cross(qt, stress) * self.l0 + _cross(Jwe, w) + Jwe * rate
        Qn = _next(Q)
        c = 0.5 * (Q * Qn).sum((0, 1)) - (0.5 + 1e-10)
        c = torch.where(V, c, 0.5)
        theta = torch.acos(c)
        st = 0.5 * theta / torch.sin(theta + 1e-14) / self.D0
        turn = torch.stack([_dot(Q[2], Qn[1]) - _dot(Q[1], Qn[2]), _dot(Q[0], Qn[2]) - _dot(Q[2], Qn[0]),
                            _dot(Q[1], Qn[0]) - _dot(Q[0], Qn[1])])
        kappa = st * turn
        eps = 0.5 * (l + _next(l)) / self.D0
        couple = self.B * (kappa - self.kap0)
        g = torch.where(V, couple / eps ** 3, zero)
        h = torch.where(V, _cross(kappa, couple) * self.D0 / eps ** 3, zero)
        T = T + g - _before(g) * self.not_first + 0.5 * (h + _before(h) * self.not_first)
        if self.w["explicit"]:
            T = T - 0.5 * (self.mass + _next(self.mass)) * self.w["explicit"] * w
        if self.contact is not None:
            cf, ct = self.contact.loads(x_rate)
            F = F + 0.5 * cf + 0.5 * _before(cf) * self.not_first
            T = T + (Q * ct[None]).sum(1)
        if self.joints:
            jf, jt = torch.zeros_like(x), torch.zeros_like(x)
            d = x[:, self.jb] - x[:, self.ja + 1]
            jf.index_add_(1, self.ja + 1, self.jk * d)
            jf.index_add_(1, self.jb, -self.jk * d)
            arm = x[:, self.jb + 1] - x[:, self.jb]
            tau = _cross(arm, -self.jrot * _dot(arm, self.jn) * self.jn)
            jt.index_add_(1, self.ja, -tau)
            jt.index_add_(1, self.jb, tau)
            F, T = F + jf, T + (Q * jt[None]).sum(1)
        if self.torque is not None:
            T = T + (Q * self.torque[None]).sum(1)
        self.v = self.v + dt * F / self.mass
        self.omega = torch.where(E, w + dt * T / self.J * e, zero)
        self.v = torch.where(self.clamped, zero, self.v)
        self.omega = torch.where(self.clamped, zero, self.omega)
        if self.w["damper"] is not None:
            nu_t, nu_r = self.w["damper"]
            self.v = self.v * math.exp(-nu_t * damper_dt)
            self.omega = self.omega * torch.exp(-nu_r * self.element_mass * damper_dt * e / self.J)

    def step(self, stepper):
        dt = self.dt
        if stepper == "position_verlet":
            parts = [(0.5, 1.0, 0.5, 1.0)]
        elif stepper == "velocity_verlet":
            parts = [(0.0, 0.5, 1.0, 1.0), (0.0, 0.5, 0.0, 1.0)]
        else:
            xi, lam, chi = 0.1786178958448091, -0.2123418310626054, -0.06626458266981849
            k = 0.5 * (1.0 - 2.0 * lam)
            parts = [(xi, k, 0.0, k), (chi, lam, 0.0, lam), (1.0 - 2.0 * (chi + xi), lam, 0.0, lam), (chi, k, xi, k)]
        for before, kick, after, damper in parts:
            if before:
                self.drift(before * dt)
            self.clamp()
            self.kick(kick * dt, damper * dt, dt)
            if after:
                self.drift(after * dt)

    def state(self):
        Q = self.Q.reshape(9, -1)
        return {"Position": self.x.cpu(), "Velocity": self.v.cpu(), "Director": Q.cpu(),
                "AngularVelocity": self.omega.cpu()}


class _Contact:
    """Spring-dashpot loads between capsules (one per element), and between capsules and the walls."""

    def __init__(self, plain, dev):
        m = plain.w["contact"]
        self.p = plain
        self.k, self.cn, self.ct = 0.5 * m.stiffness, 0.5 * m.normal_damping, 0.5 * m.tangential_damping
        self.mu = 2.0 * m.dynamic_friction
        self.ids = torch.nonzero(plain.E).squeeze(1)
        self.planes = [(torch.tensor(p, dtype=torch.float64, device=dev)[:, None],
                        torch.tensor(n, dtype=torch.float64, device=dev)[:, None]) for p, n in plain.w["planes"]]
        self.force = None

    def loads(self, dt):
        p, ids = self.p, self.ids
        a, b = p.x[:, ids], p.x[:, ids + 1]
        dx = b - a
        length = dx.square().sum(0).sqrt()
        u = dx / length
        radius = (p.volume[ids] / (math.pi * length)).sqrt()
        centre = 0.5 * (a + b)
        vel = (p.mass[ids] * p.v[:, ids] + p.mass[ids + 1] * p.v[:, ids + 1]) / (p.mass[ids] + p.mass[ids + 1])
        # the capsule's frame: the axis as third row, the others from a fixed direction
        guess = torch.tensor([0.8, 0.6, 0.0], dtype=torch.float64, device=u.device)[:, None].expand_as(u)
        other = torch.tensor([0.6, -0.8, 0.0], dtype=torch.float64, device=u.device)[:, None].expand_as(u)
        v2 = _cross(_cross(u, guess), u)
        guess = torch.where(_dot(v2, v2) < 1e-8, other, guess)
        v3 = _cross(u, guess)
        v2 = _cross(v3, u)
        r0, r1 = v2 / v2.square().sum(0).sqrt(), v3 / v3.square().sum(0).sqrt()
        om = p.omega[:, ids]
        spin = r0 * om[0] + r1 * om[1] + u * om[2]
        F, T = torch.zeros_like(centre), torch.zeros_like(centre)
        i, j = self.pairs(centre, u, length, radius)
        up = 0.5 * length * u
        on_i, on_j = _closest(centre + up, centre - up, i, j)
        normal = on_i - on_j
        far = normal.square().sum(0).sqrt()
        gap = far - radius[i] - radius[j]
        hit = (far >= 1e-8) & (gap < -1e-8)
        i, j, on_j, normal, far, gap = i[hit], j[hit], on_j[:, hit], normal[:, hit], far[hit], gap[hit]
        normal = normal / far
        at = on_j + (radius[j] + 0.5 * gap) * normal
        rel = vel[:, i] + _cross(spin[:, i], at - centre[:, i]) - vel[:, j] - _cross(spin[:, j], at - centre[:, j])
        net = self.spring(gap, normal, rel)
        F.index_add_(1, i, net)
        F.index_add_(1, j, -net)
        T.index_add_(1, i, _cross(at - centre[:, i], net))
        T.index_add_(1, j, -_cross(at - centre[:, j], net))
        for point, normal in self.planes:
            for sign in (1.0, -1.0):
                end = centre + sign * up
                gap = _dot(normal, end - point).abs() - radius
                h = torch.nonzero(gap < -1e-8).squeeze(1)
                at = end[:, h] - (radius[h] + gap[h]) * normal
                net = self.spring(gap[h], normal.expand(3, len(h)), vel[:, h] + _cross(spin[:, h], at - centre[:, h]))
                F.index_add_(1, h, net)
                T.index_add_(1, h, _cross(at - centre[:, h], net))
        cf, ct = torch.zeros_like(p.x), torch.zeros_like(p.x)
        cf[:, ids], ct[:, ids] = F, T
        self.force = cf
        return cf, ct

    def spring(self, gap, normal, rel):
        approach = -_dot(normal, rel)
        tangential = -rel - approach * normal
        slip = tangential.square().sum(0).sqrt()
        fn = torch.clamp(-self.k * gap + self.cn * approach, min=0.0)
        ft = torch.minimum(self.ct * slip, self.mu * fn)
        return fn * normal + ft * tangential / torch.where(slip > 0, slip, 1.0)

    def pairs(self, centre, u, length, radius):
        """Pairs i < j whose bounding boxes overlap, found by a grid of cells."""
        reach = (u * length).abs() * 0.5 + radius + 1e-8
        lo, hi = centre - reach, centre + reach
        cell = (2.0 * reach).max() * 1.000001
        c = torch.floor((lo - lo.amin(1, keepdim=True)) / cell).long() + 1
        across = c.amax(1) + 2
        key = (c[0] * across[1] + c[1]) * across[2] + c[2]
        order = torch.argsort(key)
        sorted_key = key[order]
        out_i, out_j = [], []
        n = torch.arange(len(key), device=key.device)
        for ox in (-1, 0, 1):
            for oy in (-1, 0, 1):
                for oz in (-1, 0, 1):
                    want = ((c[0] + ox) * across[1] + c[1] + oy) * across[2] + c[2] + oz
                    start = torch.searchsorted(sorted_key, want)
                    count = torch.searchsorted(sorted_key, want, right=True) - start
                    i = torch.repeat_interleave(n, count)
                    shift = torch.repeat_interleave(start - (torch.cumsum(count, 0) - count), count)
                    j = order[shift + torch.arange(len(i), device=i.device)]
                    keep = (i < j) & (lo[:, i] <= hi[:, j]).all(0) & (hi[:, i] >= lo[:, j]).all(0)
                    out_i.append(i[keep])
                    out_j.append(j[keep])
        return torch.cat(out_i), torch.cat(out_j)


def _closest(first, second, i, j):
    """Closest points of the segments i and j (ends `first` and `second`), region by region as the collision system
    defines them: its tolerance on the projections (1e-8 m^2) decides which region a pair falls into."""
    a1, a2, b1, b2 = first[:, i], second[:, i], first[:, j], second[:, j]
    a, b, tol = a2 - a1, b2 - b1, 1e-8
    la, lb, ab = _dot(a, a), _dot(b, b), _dot(a, b)
    r = {(p, q): y - x for p, x in ((1, a1), (2, a2)) for q, y in ((1, b1), (2, b2))}
    da = {k: _dot(a, v) for k, v in r.items()}
    db = {k: _dot(b, v) for k, v in r.items()}
    det = la * lb - ab * ab
    on_a = a1 + (lb * da[1, 1] - ab * db[1, 1]) / det * a
    on_b = b1 + (ab * da[1, 1] - la * db[1, 1]) / det * b
    k3, k4 = da[1, 1] / la * a, da[1, 2] / la * a
    k1, k2 = -db[1, 1] / lb * b, -db[2, 1] / lb * b
    regions = [
        ((da[1, 1] <= 0) & (db[1, 1] >= 0), a1, b1),
        ((da[1, 2] <= 0) & (db[1, 2] <= 0), a1, b2),
        ((da[2, 1] >= 0) & (db[2, 1] >= 0), a2, b1),
        ((da[2, 2] >= 0) & (db[2, 2] <= 0), a2, b2),
        ((da[1, 1] >= -tol) & (da[2, 1] <= tol) & (_dot(b, r[1, 1] - k3) >= -tol), a1 + k3, b1),
        ((da[1, 2] >= -tol) & (da[2, 2] <= tol) & (_dot(b, r[1, 2] - k4) <= tol), a1 + k4, b2),
        ((db[1, 1] <= tol) & (db[1, 2] >= -tol) & (_dot(a, -r[1, 1] - k1) >= -tol), a1, b1 + k1),
        ((db[2, 1] <= tol) & (db[2, 2] >= -tol) & (_dot(a, -r[2, 1] - k2) <= tol), a2, b1 + k2),
    ]
    for here, x, y in reversed(regions):
        on_a, on_b = torch.where(here, x, on_a), torch.where(here, y, on_b)
    return on_a, on_b


def exact(case, seed):
    plain = _Plain(case, _describe(case, seed))
    stepper = case.get("stepper", "position_verlet")
    for _ in range(case["steps"] * case.get("calls", 1)):
        plain.step(stepper)
    out = plain.state()
    if case["kind"] == "contact":
        out["ContactForce"] = plain.contact.force.cpu()
    if case["kind"] == "serve":  # results hold elements only where the rod has them
        keep = torch.as_tensor(_masks(_describe(case, seed))["element"])
        for name in ("Director", "AngularVelocity"):
            out[name] = out[name][:, keep]
    return out
