"""The work that users of this framework have it do, as timed cases.

A case is a dict of plain values; its "kind" says which public entry points a
pass goes through:

  steps    a time loop through the reference-shaped API: ParticleArray.set of
           the fluid's state, `steps` Integrator.integrate calls (or one
           Solver.solve), ParticleArray.get of the results
  batch    many independent scenes on one Engine: imports, step_graphed
  field    one evaluation of a 3D scene on an Engine: cells, SPHRho + Tait,
           SPHPressureGradient
  calcs    SPHCalc.sph function by function (no integrator), on particles of
           varying smoothing length
  rollout  a differentiable rollout, forward and backward

Every pass starts from the state's own inputs, so passes are alike.  Inputs
are seeded particle sets: a lattice jittered by a few per cent of its spacing
with a smooth velocity field that has the particles cross the neighbour
lists' skin at the rate a running simulation does.
"""
import math

import numpy as np
import torch

RADIUS = {"cubic": 2.0, "quintic": 3.0, "wendland": 2.0}
DEFAULT_SHAPE = {"stencil": 1, "lanes": 1, "pair_block": 128, "list_batch": 4}


# ------------------------------------------------------------------- cases
def listed():
    return [
        # The smallest call: a host program that owns numpy arrays and drives
        # one step at a time (set, integrate, get), in the default precision.
        # Launches, copies and host work count.
        dict(name="drop_1k_hostloop_fp64", kind="steps", problem="drop", n=1257, precision="fp64",
             scheme="summation", integrator="pc", kernel="cubic", variable_h=False, steps=1,
             drive="host", **DEFAULT_SHAPE),
        # The reference's elliptical drop as a whole run: Solver.solve, 100
        # steps of fixed dt, float64, every default.
        dict(name="drop_5k_solve_fp64", kind="steps", problem="drop", n=5025, precision="fp64",
             scheme="summation", integrator="pc", kernel="cubic", variable_h=False, steps=100,
             drive="solve", **DEFAULT_SHAPE),
        # A higher-order integrator and the wide kernel (support 3h, more than
        # twice the neighbours) on a drop of ordinary size.
        dict(name="drop_50k_rk4_quintic_fp32c", kind="steps", problem="drop", n=50331,
             precision="fp32c", scheme="summation", integrator="rk4", kernel="quintic",
             variable_h=False, steps=5, drive="device", **DEFAULT_SHAPE),
        # The headline workload: the 2D dam break at dx = 0.0025 with the CFL
        # time step, on the launch shape that the autotuner picks for it.
        dict(name="dam_332k_fp32c", kind="steps", problem="dam", n=320000, precision="fp32c",
             scheme="summation", integrator="pc", kernel="cubic", variable_h=False, steps=20,
             drive="device", stencil=2, lanes=1, pair_block=256, list_batch=2),
        # The dam break in float64, the precision a ParticleArray has unless
        # it asks for another, at half the resolution.
        dict(name="dam_83k_fp64", kind="steps", problem="dam", n=80000, precision="fp64",
             scheme="summation", integrator="pc", kernel="cubic", variable_h=False, steps=10,
             drive="device", **DEFAULT_SHAPE),
        # The reference's own dam-break scheme: continuity equation on fluid
        # and walls, XSPH; a spacing that divides nothing evenly.
        dict(name="dam_continuity_146k_fp32c", kind="steps", problem="dam", n=146000,
             precision="fp32c", scheme="continuity", integrator="pc", kernel="cubic",
             variable_h=False, steps=10, drive="device", **DEFAULT_SHAPE),
        # Many scenes of uneven size in one launch per stage (ensembles).
        dict(name="drops256_fp32c", kind="batch", scenes=256, n_lo=1000, n_hi=20000,
             precision="fp32c", steps=4, stencil=1, lanes=1, pair_block=128, list_batch=4),
        # 3D: one evaluation of density and pressure gradient on new
        # positions, as a post-processing or driving program asks for it.
        dict(name="lattice_2m_fp32c", kind="field", n=128, precision="fp32c", stencil=2, lanes=1,
             pair_block=128),
        dict(name="lattice_300k_fp64", kind="field", n=67, precision="fp64", stencil=2, lanes=2,
             pair_block=128),
        # Reverse mode through a rollout (fitting initial velocities).
        dict(name="rollout_20k", kind="rollout", n=20081, steps=40, every=20),
        # The function API on its own, symmetric neighbours and averaged
        # kernels over a varying smoothing length, float64.
        dict(name="calcs_varh_60k_fp64", kind="calcs", n=60000, precision="fp64", hks=True),
        # A 3D time loop of ordinary size on every default.
        dict(name="cube_64k_fp32c", kind="steps", problem="cube", n=64000, precision="fp32c",
             scheme="summation", integrator="pc", kernel="cubic", variable_h=False, steps=10,
             drive="device", **DEFAULT_SHAPE),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges (the largest listed case bounds the cost)."""
    kind = rng.choice(["steps", "steps", "steps", "steps", "batch", "field", "calcs", "rollout"])
    precision = rng.choice(["fp64", "fp32c"])
    shape = rng.choice([DEFAULT_SHAPE, DEFAULT_SHAPE,
                        dict(stencil=rng.choice([1, 2]), lanes=rng.choice([1, 2, 4]),
                             pair_block=rng.choice([64, 128, 256]),
                             list_batch=rng.choice([2, 4]))])
    if kind == "steps":
        scheme = rng.choice(["summation", "summation", "continuity"])
        integrator = rng.choice(["pc", "pc", "pc", "euler", "rk2", "rk4"])
        variable_h = rng.random() < 0.2
        problem = rng.choice(["drop", "drop", "dam", "dam", "cube"])
        kernel = "cubic"
        if problem == "drop":
            n = _log(rng, 1200, 100000)
            kernel = rng.choice(["cubic", "cubic", "quintic", "wendland"])
        else:
            n = _log(rng, 5000, 320000 if problem == "dam" else 80000)
        drive = rng.choice(["device", "device", "host", "solve"])
        if problem == "dam" and drive == "solve":
            drive = "device"
        steps = rng.randint(1, 20) if n < 100000 else rng.randint(1, 8)
        return dict(kind=kind, problem=problem, n=n, precision=precision, scheme=scheme,
                    integrator=integrator, kernel=kernel, variable_h=variable_h, steps=steps,
                    drive=drive, **shape)
    if kind == "batch":
        lo = _log(rng, 300, 3000)
        return dict(kind=kind, scenes=_log(rng, 2, 256), n_lo=lo, n_hi=lo * rng.randint(2, 6),
                    precision=precision, steps=rng.randint(1, 4), **shape)
    if kind == "field":
        return dict(kind=kind, n=_log(rng, 11, 100 if precision == "fp32c" else 72),
                    precision=precision, stencil=rng.choice([1, 2]), lanes=rng.choice([1, 2]),
                    pair_block=rng.choice([64, 128, 256]))
    if kind == "calcs":
        return dict(kind=kind, n=_log(rng, 1000, 100000), precision=precision,
                    hks=rng.random() < 0.5)
    return dict(kind=kind, n=_log(rng, 1000, 25000), steps=rng.randint(5, 40),
                every=rng.choice([5, 10, 20]))


# ------------------------------------------------------------------ inputs
def _lattice_density(kernel, h_fac, dx):
    """Density that the smoothing sum gives inside a square lattice of
    spacing dx with m = dx^2 (the reference's quintic and Wendland kernels
    are not normalised to 1; a run of theirs takes this as rest density)."""
    i = np.arange(-8, 9)
    x, y = np.meshgrid(i, i)
    q = torch.as_tensor(np.sqrt(x * x + y * y) / h_fac)
    return float(_w(kernel, 2, q * (h_fac * dx), torch.tensor(h_fac * dx, dtype=q.dtype)).sum()
                 * dx * dx)


def _drop(n, rng, dx=None, scale=100.0, kernel="cubic", variable_h=False):
    """Elliptical drop: unit disc, u = -s x, v = s y; about n particles."""
    dx = math.sqrt(math.pi / n) if dx is None else dx
    g = np.arange(-1.0, 1.0 + 1e-4, dx)
    x, y = (c.ravel() for c in np.meshgrid(g, g, indexing="ij"))
    keep = np.sqrt(x * x + y * y) <= 1.0 + 1e-10
    x, y = x[keep], y[keep]
    n = len(x)
    x = x + rng.uniform(-0.02, 0.02, n) * dx
    y = y + rng.uniform(-0.02, 0.02, n) * dx
    s = scale * rng.uniform(0.8, 1.2)
    h = np.full(n, 1.3 * dx)
    if variable_h:
        h *= 1.0 + 0.1 * np.sin(3.0 * x) * np.cos(2.0 * y)
    rho0 = 1.0 if kernel == "cubic" else _lattice_density(kernel, 1.3, dx)
    fluid = dict(x=x, y=y, u=-s * x + rng.normal(0, 0.5, n), v=s * y + rng.normal(0, 0.5, n),
                 m=np.full(n, dx * dx), h=h, rho=np.full(n, rho0), p=np.zeros(n),
                 cs=np.full(n, 1400.0))
    return [fluid], dict(c0=1400.0, rho0=rho0, gamma=7.0, alpha=0.1, beta=0.0, eta=0.1, gy=0.0,
                         cfl=0.0, dt=1e-5 * dx / 0.025)


def _dam(n, rng, variable_h=False):
    """2D dam break: a 1 x 2 column of about n particles in a 4 x 3 tank with
    three layers of fixed walls, in the collapsing flow u = a x, v = -a y."""
    dx = 1.0 / round(math.sqrt(n / 2.0))
    fx, fy = (np.arange(int(round(e / dx))) + 0.5 for e in (1.0, 2.0))
    x, y = (c.ravel() * dx for c in np.meshgrid(fx, fy, indexing="ij"))
    n = len(x)
    x = x + rng.uniform(-0.02, 0.02, n) * dx
    y = y + rng.uniform(-0.02, 0.02, n) * dx
    a = 1.5 * rng.uniform(0.8, 1.2)
    h0 = 1.3 * dx
    wx, wy = [], []
    across, up = int(round(4.0 / dx)), int(round(3.0 / dx))
    for k in range(3):
        off = (k + 0.5) * dx
        xb = (np.arange(-3, across + 3) + 0.5) * dx
        yw = (np.arange(up) + 0.5) * dx
        wx += [xb, np.full(up, -off), np.full(up, across * dx + off)]
        wy += [np.full(len(xb), -off), yw, yw]
    wx, wy = np.concatenate(wx), np.concatenate(wy)
    c0 = 10.0 * math.sqrt(2 * 9.81 * 2.0)

    def array(x, y, u, v):
        n = len(x)
        h = np.full(n, h0)
        if variable_h:
            h = h0 * (1.0 + 0.1 * np.sin(3.0 * x) * np.cos(2.0 * y))
        return dict(x=x, y=y, u=u, v=v, m=np.full(n, 1000.0 * dx * dx), h=h,
                    rho=np.full(n, 1000.0), p=np.zeros(n), cs=np.full(n, c0))
    fluid = array(x, y, a * x + rng.normal(0, 0.01, n), -a * y + rng.normal(0, 0.01, n))
    wall = array(wx, wy, np.zeros(len(wx)), np.zeros(len(wx)))
    return [fluid, wall], dict(c0=c0, rho0=1000.0, gamma=7.0, alpha=0.1, beta=0.0, eta=0.1,
                               gy=-9.81, cfl=0.3, dt=1e-4)


def _lattice3(n, rng):
    """n^3 lattice of the unit cube, every point jittered by up to 0.2 dx."""
    dx = 1.0 / n
    c = (np.arange(n) + 0.5) * dx
    x, y, z = (g.ravel() + rng.uniform(-0.2, 0.2, n ** 3) * dx
               for g in np.meshgrid(c, c, c, indexing="ij"))
    one = np.ones(n ** 3)
    return dict(x=x, y=y, z=z, u=0 * one, v=0 * one, w=0 * one, m=dx ** 3 * one,
                h=1.2 * dx * one, rho=one, p=0 * one, cs=10.0 * one)


def _cube(n, rng, variable_h=False):
    """A free cube of about n particles stretching along z: u = s x / 2,
    v = s y / 2, w = -s z about its centre."""
    n1 = round(n ** (1.0 / 3.0))
    dx = 1.0 / n1
    c = (np.arange(n1) + 0.5) * dx - 0.5
    x, y, z = (g.ravel() + rng.uniform(-0.02, 0.02, n1 ** 3) * dx
               for g in np.meshgrid(c, c, c, indexing="ij"))
    n = n1 ** 3
    s = 4.0 * rng.uniform(0.8, 1.2)
    h = np.full(n, 1.2 * dx)
    if variable_h:
        h *= 1.0 + 0.1 * np.sin(3.0 * x) * np.cos(2.0 * y)
    u, v, w = (f * s * g + rng.normal(0, 0.01, n) for f, g in ((0.5, x), (0.5, y), (-1.0, z)))
    fluid = dict(x=x, y=y, z=z, u=u, v=v, w=w, m=np.full(n, dx ** 3), h=h, rho=np.ones(n),
                 p=np.zeros(n), cs=np.full(n, 10.0))
    return [fluid], dict(c0=10.0, rho0=1.0, gamma=7.0, alpha=0.1, beta=0.0, eta=0.1, gy=0.0,
                         cfl=0.0, dt=0.2 * 1.2 * dx / 10.0)


def _scenes(case, rng):
    out = []
    sizes = np.random.default_rng(case["n_lo"]).uniform(case["n_lo"], case["n_hi"],
                                                        case["scenes"])
    for n in sizes:
        out.append(_drop(n, rng, scale=rng.uniform(50.0, 150.0)))
    return out


def _inputs(case, seed):
    rng = np.random.default_rng([seed, 20])
    kind = case["kind"]
    if kind == "steps" and case["problem"] == "drop":
        return _drop(case["n"], rng, kernel=case["kernel"], variable_h=case["variable_h"])
    if kind == "steps":
        make = {"dam": _dam, "cube": _cube}[case["problem"]]
        return make(case["n"], rng, case["variable_h"])
    if kind == "batch":
        return _scenes(case, rng)
    if kind == "calcs":
        arrays, p = _drop(case["n"], rng, variable_h=True)
        return arrays, p
    if kind == "rollout":
        arrays, p = _drop(case["n"], rng)
        return arrays, dict(p, dt=5e-6 * math.sqrt(math.pi / case["n"]) / 0.025)
    return _lattice3(case["n"], rng)


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _dev(a):
    return torch.as_tensor(a, dtype=torch.float64, device=_device())


# ----------------------------------------------------------------- prepare
def prepare(case, seed):
    return {"steps": _prepare_steps, "batch": _prepare_batch, "field": _prepare_field,
            "calcs": _prepare_calcs, "rollout": _prepare_rollout}[case["kind"]](case, seed)


def _particle_arrays(case, arrays):
    from pysph_b200.base import api as base
    from pysph_b200.base.particle_types import ParticleType
    cl = "single" if case["precision"] == "fp32c" else "double"
    types = (ParticleType.Fluid, ParticleType.Solid)
    return [base.get_particle_array(name=name, type=t, cl_precision=cl, **a)
            for name, t, a in zip(("fluid", "wall"), types, arrays)]


def _prepare_steps(case, seed):
    from pysph_b200.base import api as base
    from pysph_b200.base import kernels
    from pysph_b200.base.particle_types import ParticleType
    from pysph_b200.solver import api as solver
    from pysph_b200.sph import api as sph
    arrays, p = _inputs(case, seed)
    pas = _particle_arrays(case, arrays)
    particles = base.Particles(pas, variable_h=case["variable_h"])
    particles.engine_options = {k: case[k] for k in DEFAULT_SHAPE}
    Fluid, Solid = ParticleType.Fluid, ParticleType.Solid
    every = [Fluid, Solid] if len(pas) > 1 else [Fluid]
    dim = 3 if case["problem"] == "cube" else 2
    pos, vel = ["x", "y", "z"][:dim], ["u", "v", "w"][:dim]
    types = {"pc": solver.PredictorCorrectorIntegrator, "euler": solver.EulerIntegrator,
             "rk2": solver.RK2Integrator, "rk4": solver.RK4Integrator}
    kernel = {"cubic": kernels.CubicSplineKernel, "quintic": kernels.QuinticSplineKernel,
              "wendland": kernels.WendlandQuinticSplineKernel}[case["kernel"]](dim=dim)
    s = solver.Solver(dim=dim, integrator_type=types[case["integrator"]], kernel=kernel)
    s.dump = False
    hks = case["variable_h"]
    tait = solver.SPHOperation(sph.TaitEquation.withargs(co=p["c0"], ro=p["rho0"]),
                               on_types=every, updates=["p", "cs"], id="eos")
    if case["scheme"] == "summation":
        s.add_operation(solver.SPHOperation(sph.SPHRho.withargs(hks=hks), on_types=every,
                                            from_types=every, updates=["rho"], id="sd"))
        s.add_operation(tait)
    else:
        s.add_operation(tait)
        s.add_operation(solver.SPHIntegration(sph.SPHDensityRate.withargs(hks=hks),
                                              on_types=every, from_types=every,
                                              updates=["rho"], id="rate"))
    s.add_operation(solver.SPHIntegration(
        sph.MomentumEquation.withargs(alpha=p["alpha"], beta=p["beta"], hks=hks),
        on_types=[Fluid], from_types=every, updates=vel, id="mom"))
    if p["gy"]:
        s.add_operation(solver.SPHIntegration(sph.GravityForce.withargs(gy=p["gy"]),
                                              on_types=[Fluid], updates=["u", "v"], id="grav"))
    s.add_operation_step([Fluid])
    if case["scheme"] == "continuity":
        s.add_operation_xsph(0.5, hks=hks)
    s.set_time_step(p["dt"])
    s.setup(particles)
    plan = s.integrator.plan
    eng = particles.session(dim=plan.dim, scheme=plan.scheme, params=plan.params,
                            kernel=plan.kernel).engine
    if p["cfl"]:
        eng.update_params(cfl=p["cfl"], dt_initial=p["dt"])
        plan.params = eng.params[0]
    names = pos + vel + (["rho"] if case["scheme"] == "continuity" else [])
    start = {n: torch.as_tensor(arrays[0][n]) for n in names}
    state = dict(case=case, solver=s, arrays=pas, params=p, outputs=pos + vel + ["rho", "p"])
    if case["drive"] == "host":
        pin = (lambda t: t.pin_memory()) if torch.cuda.is_available() else (lambda t: t)
        state["start"] = {n: pin(t).numpy() for n, t in start.items()}
        state["host"] = {n: pin(torch.empty(len(arrays[0]["x"]), dtype=torch.float64))
                         for n in state["outputs"]}
    else:
        state["start"] = {n: t.to(_device()) for n, t in start.items()}
    if case["scheme"] == "continuity" and len(pas) > 1:
        state["wall_rho"] = _dev(arrays[1]["rho"])
    return state


def _engine_scheme(num_arrays=1):
    from pysph_b200.engine import fluid_scheme
    return fluid_scheme(num_arrays)


def _engine_params(p):
    return dict(c0=p["c0"], rho0=p["rho0"], gamma=p["gamma"], alpha=p["alpha"], beta=p["beta"],
                eta=p["eta"], dt=p["dt"])


def _prepare_batch(case, seed):
    from pysph_b200.engine import Engine
    scenes = _inputs(case, seed)
    eng = Engine([(a, _engine_params(p)) for a, p in scenes], _engine_scheme(), dim=2,
                 precision=case["precision"], **{k: case[k] for k in DEFAULT_SHAPE})
    names = ("x", "y", "u", "v")
    start = {n: _dev(np.concatenate([a[0][n] for a, _ in scenes])) for n in names}
    out = {n: torch.empty_like(start["x"]) for n in names + ("rho", "p")}
    return dict(case=case, engine=eng, start=start, out=out)


def _prepare_field(case, seed):
    from pysph_b200.engine import Engine
    a = _inputs(case, seed)
    eng = Engine([([a], dict(c0=10.0, rho0=1.0, alpha=0.0, beta=0.0))], _engine_scheme(), dim=3,
                 precision=case["precision"], stencil=case["stencil"], lanes=case["lanes"],
                 pair_block=case["pair_block"], step_lists=False)
    return dict(case=case, engine=eng, start={c: _dev(a[c]) for c in "xyz"})


def _prepare_calcs(case, seed):
    from pysph_b200.base import api as base
    from pysph_b200.base import kernels
    from pysph_b200.base.particle_types import ParticleType
    from pysph_b200.solver import api as solver
    from pysph_b200.sph import api as sph
    arrays, p = _inputs(case, seed)
    pa, = _particle_arrays(case, arrays)
    particles = base.Particles([pa], variable_h=True)
    Fluid = ParticleType.Fluid
    ops = [solver.SPHOperation(sph.SPHRho.withargs(hks=case["hks"]), on_types=[Fluid],
                               from_types=[Fluid], updates=["rho"], id="sd"),
           solver.SPHOperation(sph.TaitEquation.withargs(co=p["c0"], ro=p["rho0"]),
                               on_types=[Fluid], updates=["p", "cs"], id="eos"),
           solver.SPHOperation(sph.MomentumEquation.withargs(alpha=p["alpha"], beta=p["beta"],
                                                             hks=case["hks"]),
                               on_types=[Fluid], from_types=[Fluid], updates=["ax", "ay"],
                               id="mom")]
    kernel = kernels.CubicSplineKernel(dim=2)
    calcs = [c for op in ops for c in op.get_calcs(particles, kernel)]
    for n in ("ax", "ay"):
        pa.add_property({"name": n})
    start = {n: _dev(arrays[0][n]) for n in ("x", "y", "u", "v")}
    return dict(case=case, array=pa, calcs=calcs, start=start)


def _rollout_target(arrays, p, case):
    a = arrays[0]
    t = case["steps"] * p["dt"]
    return np.stack([a["x"] + 1.1 * t * a["u"], a["y"] + 1.1 * t * a["v"]])


def _prepare_rollout(case, seed):
    from pysph_b200.adjoint import Rollout
    arrays, p = _inputs(case, seed)
    r = Rollout(arrays, _engine_params(p), _engine_scheme(), dim=2, dt=p["dt"],
                steps=case["steps"], checkpoint_every=case["every"])
    return dict(case=case, rollout=r, v0=_dev(np.stack([arrays[0]["u"], arrays[0]["v"]])),
                target=_dev(_rollout_target(arrays, p, case)))


# --------------------------------------------------------------------- run
def run(state):
    return {"steps": _run_steps, "batch": _run_batch, "field": _run_field, "calcs": _run_calcs,
            "rollout": _run_rollout}[state["case"]["kind"]](state)


def _run_steps(state):
    case, s, p = state["case"], state["solver"], state["params"]
    fluid = state["arrays"][0]
    integ, names = s.integrator, state["outputs"]
    if "wall_rho" in state:
        state["arrays"][1].set(rho=state["wall_rho"])
    fluid.set(**state["start"])
    if case["drive"] == "solve":
        s.t, s.count = 0.0, 0
        s.set_final_time((case["steps"] - 0.5) * p["dt"])
        s.solve()
    for k in range(case["steps"] if case["drive"] != "solve" else 0):
        if p["cfl"]:
            integ.integrate(0.0, device_dt=True)
        else:
            integ.integrate(p["dt"])
        if case["drive"] == "host":
            # the host program reads every step's result and hands back the
            # state it read
            host = state["host"]
            for n, t in zip(names, fluid.get(*names)):
                host[n].copy_(t, non_blocking=True)
            if torch.cuda.is_available():
                torch.cuda.current_stream().synchronize()
            if k + 1 < case["steps"]:
                fluid.set(**{n: host[n].numpy() for n in state["start"]})
    if case["drive"] == "host":
        return dict(state["host"])
    out = dict(zip(names, fluid.get(*names)))
    if len(state["arrays"]) > 1:
        out["wall_rho"], out["wall_p"] = state["arrays"][1].get("rho", "p")
    return out


def _run_batch(state):
    eng, start, out = state["engine"], state["start"], state["out"]
    eng.step_graphed("pc", [(0, n, t) for n, t in start.items()])
    for _ in range(state["case"]["steps"] - 1):
        eng.step_graphed("pc")
    eng.exchange_out_many(0, list(out), list(out.values()))
    return out


def _run_field(state):
    eng = state["engine"]
    for c, t in state["start"].items():
        eng.exchange_in(0, c, t)
    eng.bin()
    eng.density(eos=True)
    # SPHPressureGradient (mode 1) over the lists the density pass recorded
    eng.momentum(gravity=False, mode=1 | (16 if eng.list_cap else 0))
    return {n: eng.get(0, n) for n in ("rho", "p", "au", "av", "aw")}


def _run_calcs(state):
    pa = state["array"]
    pa.set(**state["start"])
    for calc in state["calcs"]:
        calc.sph(*calc.updates)
    return dict(zip(("rho", "p", "cs", "ax", "ay"), pa.get("rho", "p", "cs", "ax", "ay")))


def _run_rollout(state):
    from pysph_b200.adjoint import RolloutFunction
    v = state["v0"].clone().requires_grad_(True)
    x = RolloutFunction.apply(v, state["rollout"])
    loss = ((x - state["target"]) ** 2).mean()
    loss.backward()
    return {"x": x.detach(), "grad": v.grad, "loss": loss.detach()}


# -------------------------------------------------------------------- work
def _evaluations(case):
    return case["steps"] * {"pc": 2, "euler": 1, "rk2": 2, "rk4": 4}[case.get("integrator", "pc")]


def work(case):
    """Bytes: every evaluation and integrator stage reads and writes the FP64
    state once and its density / pressure once; a call reads its inputs and
    writes its outputs.  Flops: the pair sums, per neighbour pair 16 of the
    density and 44 of the momentum equation."""
    kind = case["kind"]
    per_n3 = 4.0 / 3.0 * math.pi * 2.4 ** 3
    if kind == "field":
        n = case["n"] ** 3
        return {"bytes": n * (24 + 40), "flops": n * per_n3 * (19 + 30)}
    per_n = math.pi * (RADIUS[case.get("kernel", "cubic")] * 1.3) ** 2   # neighbours
    n = case["n"] if kind != "batch" else case["scenes"] * 0.5 * (case["n_lo"] + case["n_hi"])
    if kind == "calcs":
        return {"bytes": n * (48 + 40), "flops": n * per_n * 60}
    if kind == "rollout":
        # forward, its recompute, and per evaluation an adjoint of about
        # three times its arithmetic
        ev = 2 * case["steps"]
        return {"bytes": n * ev * 3 * (64 + 16), "flops": n * per_n * 60 * ev * 5}
    ev = _evaluations(case)
    word = 8 if case["precision"] == "fp64" else 4
    dim, pair = 2, 60
    if case.get("problem") == "cube":
        dim, per_n, pair = 3, per_n3, 72
    return {"bytes": n * (ev * (32 * dim + 4 * word) + 32 * dim + 16),
            "flops": n * per_n * pair * ev}


# --------------------------------------------------------------- tolerance
def tolerance(case):
    """About four times what a run with its pair sums in another order, or
    at float64 throughout, shows (see exact).  Pressure is the stiffest
    output: a relative density error is multiplied by gamma c0^2 / p."""
    kind = case["kind"]
    if kind == "rollout":
        return {"rel": 3e-5, "max": 3e-3}
    if case["precision"] == "fp64":
        return {"rel": 1e-9, "max": 1e-7}
    if kind in ("field", "calcs"):
        return {"rel": 1e-5, "max": 1e-3}
    return {"rel": 1e-4, "max": 1e-2}


# ------------------------------------------------------------------- exact
# The same mathematics in float64 with plain torch: neighbour pairs from a
# sorted grid, then index_add over the pair list.

def _w(kernel, dim, r, h):
    q = r / h
    if kernel == "cubic":
        fac = 10.0 / (7.0 * math.pi) / h ** 2 if dim == 2 else 1.0 / math.pi / h ** 3
        outer = 0.25 * (2 - q).clamp(min=0) ** 3
        return fac * torch.where(q <= 1, 1 - 1.5 * q * q * (1 - 0.5 * q), outer)
    if kernel == "quintic":
        t3, t2, t1 = ((k - q).clamp(min=0) ** 5 for k in (3, 2, 1))
        return 7.0 / (478.0 * math.pi) / h ** 2 * (t3 - 6 * t2 + t1)
    t = (1 - 0.5 * q).clamp(min=0) ** 4
    return 7.0 / 4.0 * math.pi / h ** 2 * t * (2 * q + 1)


def _gw(kernel, dim, r, h):
    """g with grad W = r_ab g (finite at r = 0, where r_ab = 0)."""
    r = r.clamp(min=1e-15)
    q = r / h
    if kernel == "cubic":
        fac = 10.0 / (7.0 * math.pi) / h ** 2 if dim == 2 else 1.0 / math.pi / h ** 3
        outer = -0.75 * (2 - q).clamp(min=0) ** 2 / (h * r)
        return fac * torch.where(q < 1, 3.0 * (0.75 * q - 1) / (h * h), outer)
    if kernel == "quintic":
        t3, t2, t1 = ((k - q).clamp(min=0) ** 4 for k in (3, 2, 1))
        return 7.0 / (478.0 * math.pi) / h ** 2 / (h * r) * (5 * t3 - 30 * t2 + 75 * t1)
    t = (1 - 0.5 * q).clamp(min=0) ** 3
    return 7.0 / 4.0 * math.pi / h ** 2 * (-5.0 * t) / (h * h)


def _pairs(xd, hd, xs, hs, rs, symmetric, chunk=400000):
    """(i, j): every source j with |x_i - x_j| < rs h_i (or rs h_j), i ascending."""
    with torch.no_grad():
        dim = len(xd)
        reach = float(max(hd.max(), hs.max()) if symmetric else hd.max()) * rs * (1 + 1e-9)
        lo = [float(min(a.min(), b.min())) - 1.5 * reach for a, b in zip(xd, xs)]
        cd = [((a - o) / reach).floor().to(torch.int64) for a, o in zip(xd, lo)]
        cs = [((a - o) / reach).floor().to(torch.int64) for a, o in zip(xs, lo)]
        size = [int(max(a.max(), b.max())) + 2 for a, b in zip(cd, cs)]

        def key(c):
            k = c[0]
            stride = size[0]
            for d in range(1, dim):
                k = k + stride * c[d]
                stride *= size[d]
            return k
        skey, order = torch.sort(key(cs), stable=True)
        dkey = key(cd)
        rows = [0]
        stride = size[0]
        for d in range(1, dim):
            rows = [r + stride * o for r in rows for o in (-1, 0, 1)]
            stride *= size[d]
        out_i, out_j = [], []
        for b in range(0, len(dkey), chunk):
            base = dkey[b:b + chunk]
            for row in rows:
                first = torch.searchsorted(skey, base + row - 1)
                last = torch.searchsorted(skey, base + row + 1, right=True)
                cnt = last - first
                i = torch.repeat_interleave(torch.arange(len(base), device=base.device), cnt)
                at = torch.arange(len(i), device=base.device) - (torch.cumsum(cnt, 0) - cnt)[i]
                j = order[first[i] + at]
                i = i + b
                d2 = None
                for a, c in zip(xd, xs):
                    d = a[i] - c[j]
                    d2 = d * d if d2 is None else d2 + d * d
                r = hd[i] * rs
                ok = d2 < r * r
                if symmetric:
                    r = hs[j] * rs
                    ok |= d2 < r * r
                out_i.append(i[ok])
                out_j.append(j[ok])
        return torch.cat(out_i), torch.cat(out_j)


class _Exact:
    """A scene: x, v [dim][n] and rho over all its arrays' particles in a row."""

    def __init__(self, arrays, p, dim=2, kernel="cubic", scheme="summation", symmetric=False,
                 hks=False):
        def cat(n):
            return torch.cat([_dev(a[n]) for a in arrays])
        self.dim, self.kernel, self.p, self.scheme = dim, kernel, p, scheme
        self.rs, self.symmetric, self.hks = RADIUS[kernel], symmetric, hks
        self.x = [cat(c) for c in "xyz"[:dim]]
        self.v = [cat(c) for c in "uvw"[:dim]]
        self.m, self.h, self.rho = cat("m"), cat("h"), cat("rho")
        self.nf = len(arrays[0]["x"])          # the fluid comes first and moves
        self.moves = torch.arange(len(self.m), device=self.m.device) < self.nf
        self.dtfac = self.acc2 = 0.0
        self.count = 0

    def tait(self, rho):
        p = self.p
        B = p["c0"] ** 2 * p["rho0"] / p["gamma"]
        ratio = rho / p["rho0"]
        return B * (ratio ** p["gamma"] - 1), p["c0"] * ratio ** (0.5 * (p["gamma"] - 1))

    def _kernel(self, fn, r, i, j):
        if self.hks:
            return 0.5 * (fn(self.kernel, self.dim, r, self.h[i]) +
                          fn(self.kernel, self.dim, r, self.h[j]))
        return fn(self.kernel, self.dim, r, 0.5 * (self.h[i] + self.h[j]))

    def rates(self, x, v, rho):
        """(position rate, acceleration, density rate, rho, p, cs)"""
        p, dim = self.p, self.dim
        i, j = _pairs(x, self.h, x, self.h, self.rs, self.symmetric)
        r = [c[i] - c[j] for c in x]
        r2 = sum(c * c for c in r)
        same = i == j
        dist = torch.sqrt(torch.where(same, torch.ones_like(r2), r2))
        dist = torch.where(same, torch.zeros_like(r2), dist)
        zero = torch.zeros_like(self.m)
        summed = self.scheme == "summation"
        if summed:
            rho = zero.index_add(0, i, self.m[j] * self._kernel(_w, dist, i, j))
        pres, cs = self.tait(rho)
        g = self._kernel(_gw, dist, i, j)
        dv = [c[i] - c[j] for c in v]
        dot = sum(a * b for a, b in zip(dv, r))
        drho = None if summed else zero.index_add(0, i, self.m[j] * dot * g)
        f = i < self.nf                         # the momentum equation acts on the fluid
        fi, fj, fg = i[f], j[f], g[f]
        fr, fdot, fr2 = [c[f] for c in r], dot[f], r2[f]
        hab = 0.5 * (self.h[fi] + self.h[fj])
        mu = hab * fdot / (fr2 + p["eta"] ** 2 * hab * hab)
        vis = (-p["alpha"] * 0.5 * (cs[fi] + cs[fj]) * mu + p["beta"] * mu * mu) / (
            0.5 * (rho[fi] + rho[fj]))
        t = pres[fi] / rho[fi] ** 2 + pres[fj] / rho[fj] ** 2
        t = t + torch.where(fdot < 0, vis, torch.zeros_like(vis))
        acc = [zero.index_add(0, fi, -self.m[fj] * t * fg * c) for c in fr]
        acc[1] = acc[1] + torch.where(self.moves, p["gy"], 0.0)
        if p["cfl"]:
            self.dtfac = float(mu.abs().max())
            self.acc2 = float(sum(c[:self.nf] ** 2 for c in acc).max())
        xr = [torch.where(self.moves, c, zero) for c in v]
        if not summed:
            q = f & (j < self.nf)               # XSPH from the fluid, eps = 0.5
            qi, qj = i[q], j[q]
            w = self._kernel(_w, dist[q], qi, qj)
            w = 0.5 * self.m[qj] * w / (0.5 * (rho[qi] + rho[qj]))
            xr = [a.index_add(0, qi, -w * c[q]) for a, c in zip(xr, dv)]
        return xr, acc, drho, rho, pres, cs

    def dt(self):
        p = self.p
        self.count += 1
        if not p["cfl"]:
            return p["dt"]
        h = float(self.h[:self.nf].min())
        force = p["dt"] if self.count == 1 else math.sqrt(self.acc2)
        return min(1.0, p["cfl"] * h / (p["c0"] + self.dtfac), p["cfl"] * math.sqrt(h / force))

    def step(self, integrator):
        dt = self.dt()
        x0, v0, r0 = self.x, self.v, self.rho

        def at(k, f):
            add = lambda a, b: [s + f * t for s, t in zip(a, b)]  # noqa: E731
            return add(x0, k[0]), add(v0, k[1]), r0 if k[2] is None else r0 + f * k[2]

        def rates(s):
            k = self.rates(*s)
            self.pres, self.cs, summed = k[4], k[5], k[2] is None
            if summed:
                self.summed = k[3]
            return k
        k1 = rates((x0, v0, r0))
        if integrator == "euler":
            new = at(k1, dt)
        elif integrator == "rk4":
            k2 = rates(at(k1, dt / 2))
            k3 = rates(at(k2, dt / 2))
            k4 = rates(at(k3, dt))
            mix = [None if a is None else
                   [p + 2 * q + 2 * r + s for p, q, r, s in zip(a, b, c, d)]
                   if isinstance(a, list) else a + 2 * b + 2 * c + d
                   for a, b, c, d in zip(k1[:3], k2[:3], k3[:3], k4[:3])]
            new = at(mix, dt / 6)
        else:
            # 2 (X0 + dt/2 F) - X0 of the predictor-corrector is RK2's X0 + dt F
            new = at(rates(at(k1, dt / 2)), dt)
        self.x, self.v, self.rho = new

    def outputs(self):
        f = slice(0, self.nf)
        rho = self.summed if self.scheme == "summation" else self.rho
        out = dict(zip("xyz", (c[f] for c in self.x)))
        out.update(zip("uvw", (c[f] for c in self.v)))
        out.update(rho=rho[f], p=self.pres[f])
        if self.nf < len(self.m):
            out["wall_rho"], out["wall_p"] = rho[self.nf:], self.pres[self.nf:]
        return out


def exact(case, seed):
    kind = case["kind"]
    data = _inputs(case, seed)
    if kind == "field":
        return _exact_field(data)
    if kind == "batch":
        outs = []
        for arrays, p in data:
            e = _Exact(arrays, p)
            for _ in range(case["steps"]):
                e.step("pc")
            outs.append(e.outputs())
        return {n: torch.cat([o[n] for o in outs]) for n in outs[0]}
    arrays, p = data
    if kind == "calcs":
        e = _Exact(arrays, p, symmetric=True, hks=case["hks"])
        _, acc, _, rho, pres, cs = e.rates(e.x, e.v, e.rho)
        return dict(rho=rho, p=pres, cs=cs, ax=acc[0], ay=acc[1])
    if kind == "rollout":
        e = _Exact(arrays, p)
        v0 = torch.stack(e.v).requires_grad_(True)
        e.v = [v0[0], v0[1]]
        for _ in range(case["steps"]):
            e.step("pc")
        x = torch.stack(e.x)
        loss = ((x - _dev(_rollout_target(arrays, p, case))) ** 2).mean()
        loss.backward()
        return {"x": x.detach(), "grad": v0.grad, "loss": loss.detach()}
    e = _Exact(arrays, p, dim=3 if case["problem"] == "cube" else 2, kernel=case["kernel"],
               scheme=case["scheme"],
               symmetric=case["variable_h"], hks=case["variable_h"])
    for _ in range(case["steps"]):
        e.step(case["integrator"])
    out = e.outputs()
    if case["drive"] == "host":
        out = {n: t for n, t in out.items() if not n.startswith("wall_")}
    return out


def _exact_field(a, chunk=200000):
    x, h, m = [_dev(a[c]) for c in "xyz"], _dev(a["h"]), _dev(a["m"])
    n = len(h)
    rho = torch.zeros_like(h)

    def each(fn):
        for b in range(0, n, chunk):
            s = slice(b, min(n, b + chunk))
            i, j = _pairs([c[s] for c in x], h[s], x, h, 2.0, False)
            i = i + b
            r = [c[i] - c[j] for c in x]
            fn(i, j, r, torch.sqrt(sum(c * c for c in r)))

    def density(i, j, r, dist):
        rho.index_add_(0, i, m[j] * _w("cubic", 3, dist, 0.5 * (h[i] + h[j])))
    each(density)
    pres = 100.0 / 7.0 * (rho ** 7 - 1)
    acc = [torch.zeros_like(h) for _ in x]
    t = pres / rho ** 2

    def gradient(i, j, r, dist):
        g = -m[j] * (t[i] + t[j]) * _gw("cubic", 3, dist, 0.5 * (h[i] + h[j]))
        for s, c in zip(acc, r):
            s.index_add_(0, i, g * c)
    each(gradient)
    return dict(rho=rho, p=pres, au=acc[0], av=acc[1], aw=acc[2])
