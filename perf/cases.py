"""The work a user of femorax_b200 has it do, as cases that can be timed and checked: operator
applies, explicit steps, static, Newmark and J2 Newton solves, batched and served solves, and the
multi-yield soils as material points and on the element path, each through the package's public
entry points. `listed` names the cases, `draw` gives more of the same ranges, `prepare` makes what a
program has in hand before the call, `run` is one call, `exact` the same result in plain torch.

Meshes go with a case's sizes (a program compiles its model once), the vectors, loads and strains
come from the seed."""
import functools
import math

import numpy as np
import torch

import femorax_b200 as fx
from femorax_b200 import meshes, stages

DEV = torch.device("cuda", 0)
F64 = torch.float64

# dense sand of the stored PressureDependMultiYield paths, clay of the plastic box
SAND = (2.0285423037716614, 145000.0, 314166.66666666663, 40.0, 0.1, 80.0, 0.5, 27.0, 0.03, 0.8, 5.0, 0.0, 0.0, 0.0)
CLAY = (1.8, 40500.0, 108000.0, 8.0, 0.1, 0.0, 100.0, 0.0)


def listed():
    return [
        # a small mixed-precision operator call: one FP32 apply, bound by latency
        dict(name="apply_small_f32", kind="apply", mesh="cube", nx=24, ny=21, nz=18, f32=True, mass=0.0, damping=0.0),
        # the benchmark's operator: the layered soil box of the explicit wave configuration
        dict(name="apply_layered", kind="apply", mesh="layered", nx=128, ny=128, nz=64, f32=False, mass=0.0,
             damping=0.0),
        # explicit wave propagation on a layered box of ragged size
        dict(name="explicit_layered", kind="explicit", nx=101, ny=75, nz=61, steps=48, f32=False),
        # the static configuration: a 32^3 block under a top load, Jacobi-PCG to 1e-10
        dict(name="static_cube", kind="static", nx=32, ny=32, nz=32, rtol=1e-10, mixed=False),
        # implicit dynamics with per-element moduli: FP32 CG inside FP64 refinement
        dict(name="newmark_mixed", kind="newmark", n=44, steps=2, mixed=True),
        # the effective operator of an implicit step on a distorted mesh, in the reference's arithmetic
        dict(name="general_apply", kind="apply", mesh="distorted", nx=37, ny=31, nz=43, f32=False, mass=1.6e7,
             damping=2e3),
        # the reference's benchmark model: the damped internal force of the 40^3 laminar soil column
        dict(name="column_force", kind="force", nx=40, ny=40, nz=40, mode="fast"),
        # one load step of a J2 block: Newton with the consistent tangent, Jacobi-PCG
        dict(name="j2_newton", kind="j2", nx=16, ny=16, nz=20, count=1, load=1.0),
        # the batched J2 configuration: one load step of many seeded columns and blocks at once
        dict(name="j2_batch", kind="j2", nx=8, ny=8, nz=40, count=24, load=1.0),
        # explicit shaking of a plastic clay box, material commits included
        dict(name="pimy_stage", kind="soil_stage", n=46, steps=16, corrector="fused"),
        # material points of a dense sand on cyclic shear paths
        dict(name="pdmy_points", kind="points", material="pdmy", points=300001),
        # many static solves of different sizes through one batched engine
        dict(name="engine_mixed", kind="engine", count=16, lo=10, hi=44, inner="fp32"),
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("apply", "apply", "explicit", "static", "newmark", "general", "force", "j2", "j2_batch",
                       "soil_force", "soil_stage", "points", "engine"))
    if kind == "apply":
        return dict(kind="apply", mesh=rng.choice(("layered", "cube")), nx=_size(rng, 9, 60), ny=_size(rng, 9, 60),
                    nz=_size(rng, 8, 50), f32=rng.random() < 0.5, mass=rng.choice((0.0, 1.6e7)),
                    damping=rng.choice((0.0, 2e3)))
    if kind == "explicit":
        return dict(kind="explicit", nx=_size(rng, 12, 90), ny=_size(rng, 12, 70), nz=_size(rng, 9, 60),
                    steps=rng.randint(17, 48), f32=rng.random() < 0.4)
    if kind == "static":
        return dict(kind="static", nx=_size(rng, 4, 36), ny=_size(rng, 4, 30), nz=_size(rng, 4, 30),
                    rtol=rng.choice((1e-8, 1e-10)), mixed=rng.random() < 0.3)
    if kind == "newmark":
        return dict(kind="newmark", n=_size(rng, 6, 40), steps=rng.randint(1, 3), mixed=rng.random() < 0.5)
    if kind == "general":
        return dict(kind="apply", mesh=rng.choice(("distorted", "column", "ssp")), nx=_size(rng, 4, 40),
                    ny=_size(rng, 4, 36), nz=_size(rng, 4, 40), f32=False, mass=rng.choice((0.0, 1.6e7)),
                    damping=rng.choice((0.0, 2e3)))
    if kind == "force":
        return dict(kind="force", nx=_size(rng, 5, 38), ny=_size(rng, 5, 38), nz=_size(rng, 5, 38),
                    mode=rng.choice(("fast", "exact")))
    if kind == "j2":
        return dict(kind="j2", nx=_size(rng, 1, 14), ny=_size(rng, 1, 14), nz=_size(rng, 4, 20), count=1,
                    load=round(rng.uniform(0.5, 1.1), 3))
    if kind == "j2_batch":
        return dict(kind="j2", nx=_size(rng, 1, 8), ny=_size(rng, 1, 8), nz=_size(rng, 8, 36),
                    count=rng.randint(2, 20), load=round(rng.uniform(0.5, 1.1), 3))
    if kind == "soil_force":
        return dict(kind="soil_force", material=rng.choice(("pimy", "pdmy")), nx=_size(rng, 3, 38),
                    ny=_size(rng, 3, 38), nz=_size(rng, 3, 38), corrector=rng.choice(("fused", "compacted")))
    if kind == "soil_stage":
        return dict(kind="soil_stage", n=_size(rng, 4, 40), steps=rng.randint(3, 20),
                    corrector=rng.choice(("fused", "compacted")))
    if kind == "points":
        return dict(kind="points", material=rng.choice(("pimy", "pdmy")), points=_size(rng, 100, 260000))
    return dict(kind="engine", count=rng.randint(2, 14), lo=rng.randint(4, 12), hi=rng.randint(16, 40),
                inner=rng.choice(("fp32", "fp64")))


# ---------------------------------------------------------------- models
class _Built:
    """A compiled model: the spec, the compile step's arrays and the DOF of every equation."""

    def __init__(self, spec):
        self.spec = spec
        comp = fx.Model(spec).compile()
        self.mesh = comp.mesh()
        self.eqmap = meshes.equation_map(comp)
        self.dof = comp.array("eq_dof")


def _soil_elastic(material):
    G, K = (SAND if material == "pdmy" else CLAY)[1:3]
    return 9 * K * G / (3 * K + G), (3 * K - 2 * G) / (2 * (3 * K + G))


@functools.lru_cache(maxsize=48)
def _built(kind, nx, ny, nz):
    if kind == "layered":
        return _Built(meshes.layered_box(nx, ny, nz, layers=min(8, nz), seed=0)[0])
    if kind == "cube":  # one material per element
        spec = meshes.box_model(nx, ny, nz, (0.5 * nx, 0.5 * ny, 0.5 * nz), rho=2000.0)
        g = spec.groups[0]
        E = 80e6 * np.exp(0.5 * np.random.default_rng(0).standard_normal(len(g.etags)))
        spec.groups = [meshes.Group(float(E[e]), 0.3, 2000.0, g.etags[e:e + 1], g.conn[e:e + 1])
                       for e in range(len(E))]
        return _Built(spec)
    if kind == "block":
        return _Built(meshes.box_model(nx, ny, nz, (1.0, ny / nx, nz / nx)))
    if kind == "distorted":
        spec = meshes.box_model(nx, ny, nz, (float(nx), float(ny), float(nz)), E=1.1e5, nu=0.3, rho=2.0)
        spec.rayleigh = [meshes.Rayleigh(0.6, 5.8e-4, 0.0, 0.0, spec.groups[0].etags)]
        return _Built(meshes.distort(spec, 0.2, seed=1))
    if kind in ("column", "ssp"):
        return _Built(meshes.laminar_column(nx, ny, nz, lumped=False, element=1 if kind == "ssp" else 0))
    if kind == "lumped_column":
        return _Built(meshes.laminar_column(nx, ny, nz, lumped=True))
    if kind == "j2":
        return _Built(meshes.box_model(nx, ny, nz, (0.5 * nx, 0.5 * ny, 0.5 * nz), E=80e6, nu=0.3, kind=1,
                                       sigma_y=100e3, H=4e6, hk=0.5))
    E, nu = _soil_elastic(kind)  # "pimy" or "pdmy": a box of unit elements
    rho = (SAND if kind == "pdmy" else CLAY)[0]
    return _Built(meshes.box_model(nx, ny, nz, (float(nx), float(ny), float(nz)), E=E, nu=nu, rho=rho, lumped=True))


def _engine_sizes(case):
    """Block sizes spread over [lo, hi] elements per side (over the logarithm), not quite cubes."""
    n = case["count"]
    out = []
    for i in range(n):
        s = int(round(case["lo"] * (case["hi"] / case["lo"]) ** (i / max(n - 1, 1))))
        out.append((s, max(2, s - i % 3), max(2, s + i % 2)))
    return out


def _j2_sizes(case):
    if case["count"] == 1:
        return [(case["nx"], case["ny"], case["nz"])]
    out = []
    for i in range(case["count"]):
        s = (1, 2, 4, 8)[i % 4]
        out.append((min(s, case["nx"]), min(s, case["ny"]), max(2, case["nz"] - i % 21)))
    return out


def _parts(case):
    """The compiled models of a case."""
    k = case["kind"]
    if k == "apply":
        return [_built(case["mesh"], case["nx"], case["ny"], case["nz"])]
    if k == "explicit":
        return [_built("layered", case["nx"], case["ny"], case["nz"])]
    if k == "static":
        return [_built("block", case["nx"], case["ny"], case["nz"])]
    if k == "newmark":
        return [_built("cube", case["n"], case["n"], case["n"])]
    if k == "force":
        return [_built("lumped_column", case["nx"], case["ny"], case["nz"])]
    if k == "j2":
        return [_built("j2", *s) for s in _j2_sizes(case)]
    if k == "soil_force":
        return [_built(case["material"], case["nx"], case["ny"], case["nz"])]
    if k == "soil_stage":
        return [_built("pimy", case["n"], case["n"], case["n"])]
    if k == "engine":
        return [_built("block", *s) for s in _engine_sizes(case)]
    return []


# ---------------------------------------------------------------- inputs
def _vector(seed, n, scale=1.0):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return scale * torch.randn(n, dtype=F64, device=DEV, generator=g)


def _top_load(b, seed, total):
    """A vertical and horizontal top load summing to about `total`, uneven from node to node."""
    nx, ny, nz = b.spec.grid[:3]
    rng = np.random.default_rng(seed)
    f = np.zeros(b.mesh.num_equations)
    top = np.arange((nx + 1) * (ny + 1)) + 1 + (nx + 1) * (ny + 1) * nz
    for d, share in ((2, -1.0), (0, 0.4)):
        q = b.eqmap[top, d]
        f[q[q >= 0]] = share * total / len(top) * rng.uniform(0.5, 1.5, int((q >= 0).sum()))
    return f


def _shear_load(b, seed, load):
    """The seeded J2 configuration's load: a top shear of `load` times the force that first yields
    the base in bending, or in shear where that is less."""
    nx, ny, nz, hx, hy, hz = b.spec.grid
    g = b.spec.groups[0]
    w, d, L = nx * hx, ny * hy, nz * hz
    first = min(g.sigma_y * w * w * d / (6.0 * L), 0.5 * g.sigma_y * w * d / math.sqrt(3.0))
    f, _ = stages.top_shear(b.spec, b.eqmap, 1.2 * load * first)
    return f * np.random.default_rng(seed).uniform(0.95, 1.05)


def _ground(seed, steps, dt):
    t0 = np.random.default_rng(seed).uniform(0.0, 0.1)
    return 3.0 * np.sin(2 * math.pi * 5.0 * (t0 + dt * np.arange(1, steps + 1)))


def _material(name, surfaces=20):
    if name == "pimy_points":  # a frictional sand with pressure-dependent moduli
        return fx.PressureIndependMultiYield(2.0, 60000, 150000, 5, 0.1, 30, 80, 0.5, surfaces)
    if name == "pimy":
        return fx.PressureIndependMultiYield(*CLAY, noYieldSurf=surfaces)
    return fx.PressureDependMultiYield(*SAND, noYieldSurf=surfaces, e=0.45)


def _bind(force, material):
    (force.set_pimy if material == "pimy" else force.set_pdmy)(0, _material(material))


def _position(b):
    """x and z of the node of every equation."""
    m = b.mesh
    X = m.coords.reshape(3, -1)
    node, eq = m.node.reshape(8, m.padded), m.eq.reshape(24, m.padded)
    xq, zq = np.zeros(m.num_equations), np.zeros(m.num_equations)
    for a in range(24):
        q = eq[a, :m.count]
        ok = q >= 0
        nd = node[a // 3, :m.count][ok]
        xq[q[ok]], zq[q[ok]] = X[0, nd], X[2, nd]
    return xq, zq


# ---------------------------------------------------------------- what a program has before the call
def prepare(case, seed):
    return _PREPARE[case["kind"]](case, int(seed), _parts(case))


def _prepare_apply(case, seed, parts):
    b = parts[0]
    n = b.mesh.num_equations
    x = _vector(seed, n)
    if case["f32"]:
        x = x.float()
    return dict(run=_run_apply, force=fx.InternalForce(b.mesh), x=x, y=torch.zeros_like(x),
                k=fx.OperatorCoefficients(1.0, case["damping"], case["mass"]))


def _run_apply(s):
    s["force"].apply_operator(s["k"], s["x"], s["y"])
    return s["y"]


def _prepare_force(case, seed, parts):
    b = parts[0]
    n = b.mesh.num_equations
    force = fx.InternalForce(b.mesh)
    force.set_general_mode(case["mode"])
    return dict(run=_run_force, force=force, u=_vector(seed, n, 1e-4), v=_vector(seed + 1, n, 1e-3),
                f=torch.zeros(n, dtype=F64, device=DEV))


def _run_force(s):
    s["force"].compute(s["u"], s["v"], s["f"])
    return s["f"]


def _explicit_dt(force, case):
    return 0.5 * force.min_critical_dt("ExplicitDifference")


def _prepare_explicit(case, seed, parts):
    b = parts[0]
    n = b.mesh.num_equations
    force = fx.InternalForce(b.mesh)
    t = torch.float32 if case["f32"] else F64
    dt = _explicit_dt(force, case)
    return dict(run=_run_explicit, force=force, mass=torch.as_tensor(b.mesh.lumped_mass, device=DEV).to(t), dt=dt,
                steps=case["steps"], ag=_ground(seed, case["steps"], dt), u=_vector(seed, n, 1e-4).to(t),
                vh=_vector(seed + 1, n, 1e-3).to(t), a=torch.zeros(n, dtype=t, device=DEV),
                v=torch.zeros(n, dtype=t, device=DEV))


def _run_explicit(s):
    s["force"].explicit_run(s["mass"], s["u"], s["vh"], s["a"], s["v"], s["dt"], s["steps"], ag=s["ag"], direction=0)
    return s["u"], s["vh"], s["a"], s["v"]


def _prepare_static(case, seed, parts):
    b = parts[0]
    force = fx.InternalForce(b.mesh)
    opts = fx.SolveOptions(relative_tolerance=case["rtol"])
    solver = fx.MixedPrecisionSolver(opts) if case["mixed"] else fx.ConjugateGradient(opts)
    solver.setup(fx.MatrixFreeOperator(force, fx.OperatorCoefficients()))
    return dict(run=_run_static, solver=solver, b=torch.as_tensor(_top_load(b, seed, 1e5), device=DEV),
                x=torch.zeros(b.mesh.num_equations, dtype=F64, device=DEV))


def _run_static(s):
    s["x"].zero_()
    r = s["solver"].solve(s["b"], s["x"])
    return s["x"], float(r.converged)


NEWMARK_DT = 2e-3


def _prepare_newmark(case, seed, parts):
    b = parts[0]
    n = b.mesh.num_equations
    force = fx.InternalForce(b.mesh)
    opts = fx.SolveOptions(relative_tolerance=1e-8, max_iterations=20000)
    solver = fx.MixedPrecisionSolver(opts) if case["mixed"] else fx.ConjugateGradient(opts)
    dt = NEWMARK_DT
    solver.setup(fx.MatrixFreeOperator(force, fx.OperatorCoefficients(1.0, 2.0 / dt, 4.0 / dt ** 2)))
    f, _ = stages.top_shear(b.spec, b.eqmap, 1e6)
    f = torch.as_tensor(f * np.random.default_rng(seed).uniform(0.5, 1.5, len(f)), device=DEV)
    loads = [f * math.sin(2 * math.pi * 5.0 * (i + 1) * dt) for i in range(case["steps"])]
    return dict(run=_run_newmark, solver=solver, force=force, loads=loads, dt=dt,
                uva=[torch.zeros(n, dtype=F64, device=DEV) for _ in range(3)])


def _run_newmark(s):
    for w in s["uva"]:
        w.zero_()
    for f in s["loads"]:
        s["solver"].newmark_step(f, *s["uva"], s["dt"])
        s["force"].commit_state()
    return list(s["uva"])


def _prepare_j2(case, seed, parts):
    loads = [_shear_load(b, seed + i, case["load"]) for i, b in enumerate(parts)]
    opts = fx.SolveOptions(relative_tolerance=1e-12, max_iterations=20000)
    if case["count"] == 1:
        force = fx.InternalForce(parts[0].mesh)
        solver = fx.ConjugateGradient(opts)
        solver.setup(fx.MatrixFreeOperator(force, fx.OperatorCoefficients()))
        f = torch.as_tensor(loads[0], device=DEV)
        return dict(run=_run_j2, force=force, solver=solver, f=f, u=torch.zeros_like(f))
    batch = fx.BatchedNewton([b.mesh for b in parts], opts)
    f = torch.as_tensor(batch.combine(loads), device=DEV)
    return dict(run=_run_j2_batch, batch=batch, f=f, u=torch.zeros_like(f))


def _run_j2(s):  # from the virgin state: nothing is committed, so every call is the same load step
    s["u"].zero_()
    _, r = s["solver"].newton(s["f"], s["u"], tol=1e-5)
    return s["u"], float(r.converged)


def _run_j2_batch(s):
    s["u"].zero_()
    _, r = s["batch"].step(s["f"], s["u"], tol=1e-5)
    return s["u"], float(all(x.converged for x in r))


def _prepare_soil_force(case, seed, parts):
    """A box of the soil, confined, sheared in the plastic stage and committed; the force at a
    further uneven shear."""
    b = parts[0]
    n = b.mesh.num_equations
    force = fx.InternalForce(b.mesh)
    _bind(force, case["material"])
    force.set_soil_corrector(case["corrector"])
    xq, zq = _position(b)
    zero = torch.zeros(n, dtype=F64, device=DEV)
    f = torch.zeros(n, dtype=F64, device=DEV)
    conf = np.where(b.dof == 2, -1e-4 * zq, 0.0) + np.where(b.dof == 0, -1e-4 * xq, 0.0)

    def at(gamma):
        return torch.as_tensor(conf + np.where(b.dof == 0, gamma * zq, 0.0), device=DEV)

    force.compute(at(0.0), zero, f)
    force.commit_state()
    force.set_material_stage(0, 1)
    force.compute(at(2e-4), zero, f)
    force.commit_state()
    u = at(2.7e-4) + _vector(seed, n, 1e-6)
    return dict(run=_run_force, force=force, u=u, v=zero, f=f)


def _prepare_soil_stage(case, seed, parts):
    """A clay box shaken until its lower part yields; the stage goes on from there."""
    b = parts[0]
    n = b.mesh.num_equations
    force = fx.InternalForce(b.mesh)
    _bind(force, "pimy")
    force.set_material_stage(0, 1)
    force.set_soil_corrector(case["corrector"])
    dt = 5e-4
    a0, f0 = np.random.default_rng(seed).uniform((5.0, 7.0), (6.0, 8.0))
    t = np.arange(1 << 16) * dt
    motions = fx.GroundMotions([dict(dof=0, fact=1.0, values=a0 * np.sin(2 * math.pi * f0 * t), dt=dt)])
    mass = torch.as_tensor(b.mesh.lumped_mass, device=DEV)
    u, v, a = (torch.zeros(n, dtype=F64, device=DEV) for _ in range(3))
    time, _ = force.explicit_stage("ExplicitDifference", mass, u, v, a, dt, 400, motions=motions)
    return dict(run=_run_soil_stage, force=force, motions=motions, mass=mass, uva=(u, v, a), dt=dt,
                steps=case["steps"], time=time)


def _run_soil_stage(s):
    s["time"], _ = s["force"].explicit_stage("ExplicitDifference", s["mass"], *s["uva"], s["dt"], s["steps"],
                                             time=s["time"], motions=s["motions"], resume=True)
    return s["uva"]


def _prepare_points(case, seed, parts):
    """Points of a soil confined, switched to the plastic stage and sheared twice; the update to the
    next strain of their cyclic paths."""
    n = case["points"]
    pdmy = case["material"] == "pdmy"
    m = _material("pdmy" if pdmy else "pimy_points")
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    amp = 2e-4 + ((5e-3 if pdmy else 2e-2) - 2e-4) * torch.rand(n, dtype=F64, device=DEV, generator=g)
    dirs = torch.randn(3, n, dtype=F64, device=DEV, generator=g)
    dirs /= dirs.norm(dim=0)
    conf = -2e-3 + 1.5e-3 * torch.rand(n, dtype=F64, device=DEV, generator=g)

    def strain(k):
        return torch.cat((conf.expand(3, n) / 3, amp * math.sin(2 * math.pi * k / 10) * dirs)).contiguous()

    c, t = m.initial_state(n, 0), torch.empty((m.nstate, n), dtype=F64, device=DEV)
    sig, tan = torch.empty((6, n), dtype=F64, device=DEV), torch.empty((36, n), dtype=F64, device=DEV)
    failed = torch.zeros(1, dtype=torch.int32, device=DEV)
    for stage, k in ((0, 0), (1, 0), (1, 1), (1, 2)):
        m.update(stage, c, t, strain(k), sig, tan, failed)
        c, t = t, c
    return dict(run=_run_points, m=m, c=c, t=t, eps=strain(3), sig=sig, tan=tan, failed=failed)


def _run_points(s):
    s["m"].update(1, s["c"], s["t"], s["eps"], s["sig"], s["tan"], s["failed"])
    return s["t"], s["sig"], s["tan"]


def _prepare_engine(case, seed, parts):
    opts = fx.SolveOptions(relative_tolerance=1e-8)
    capacity = sum((b.mesh.num_equations + 2047) // 2048 * 2048 for b in parts)
    tol = 1e-4 if case["inner"] == "fp32" else 1e-9
    engine = fx.BatchEngine(capacity, len(parts), options=opts, inner_tolerance=tol, inner=case["inner"])
    return dict(run=_run_engine, engine=engine, forces=[fx.InternalForce(b.mesh) for b in parts],
                b=[_top_load(b, seed + i, 1e5) for i, b in enumerate(parts)])


def _run_engine(s):
    e = s["engine"]
    slots = [e.admit(f, b) for f, b in zip(s["forces"], s["b"])]
    while e.round() > 0:
        pass
    return [e.retire(slot, len(b))[0] for slot, b in zip(slots, s["b"])]


_PREPARE = dict(apply=_prepare_apply, force=_prepare_force, explicit=_prepare_explicit, static=_prepare_static,
                newmark=_prepare_newmark, j2=_prepare_j2, soil_force=_prepare_soil_force,
                soil_stage=_prepare_soil_stage, points=_prepare_points, engine=_prepare_engine)


def run(state):
    return state["run"](state)


# ---------------------------------------------------------------- what a pass cannot do without
def _counts(parts):
    return (sum(b.mesh.num_equations for b in parts), sum(b.mesh.count for b in parts),
            sum(b.mesh.num_nodes for b in parts))


def work(case):
    """Bytes: each input read and each output written once (maps of 4 bytes per node equation and
    element parameter, coordinates and connectivity on meshes that are no grid). FLOPs: 330 per box
    element and apply, 6,000 per element of the Gauss-point form."""
    k = case["kind"]
    parts = _parts(case)
    neq, nel, nn = _counts(parts)
    w = 4 if case.get("f32") else 8
    if k == "apply" and case["mesh"] in ("layered", "cube"):
        return dict(bytes=2 * w * neq + 4 * nn + (4 if case["mesh"] == "layered" else w) * nel, flops=330 * nel)
    if k in ("apply", "force"):
        vectors = 2 if k == "apply" else 3
        return dict(bytes=8 * vectors * neq + 24 * nn + 12 * nn + 36 * nel, flops=6000 * nel)
    if k == "explicit":  # per step u, vh, a read and written, the mass read
        return dict(bytes=case["steps"] * (7 * w * neq + 4 * nn + 4 * nel), flops=case["steps"] * 350 * nel)
    if k == "static":  # iterations of Jacobi-PCG: about 7 per element along the longest side
        it = 7 * max(case["nx"], case["ny"], case["nz"])
        return dict(bytes=16 * neq + 4 * nn, flops=it * (330 * nel + 13 * neq))
    if k == "newmark":
        it = case["steps"] * 40
        return dict(bytes=case["steps"] * 72 * neq, flops=it * (330 * nel + 13 * neq))
    if k == "j2":  # Newton iterations of a plastic step times Jacobi-PCG iterations of the tallest mesh
        it = 4 * 10 * max(max(s) for s in _j2_sizes(case))
        return dict(bytes=16 * neq + 1000 * nel, flops=it * (6000 * nel + 13 * neq))
    if k == "soil_force":
        return dict(bytes=24 * neq + 8 * nel * (191 + 31 + 16) * 8 + 36 * nn, flops=8 * nel * 1500)
    if k == "soil_stage":  # the state read, its scalars written, the commit of the points that changed
        return dict(bytes=case["steps"] * (56 * neq + 8 * nel * (2 * 31 + 2 * 16) * 8), flops=case["steps"] * 8 * nel * 1500)
    if k == "points":
        state = 191 if case["material"] == "pimy" else 209
        return dict(bytes=case["points"] * 8 * (2 * state + 6 + 6 + 36), flops=case["points"] * 2000)
    return dict(bytes=sum(16 * b.mesh.num_equations for b in parts),
                flops=sum(7 * max(b.spec.grid[:3]) * (330 * b.mesh.count + 13 * b.mesh.num_equations) for b in parts))


def tolerance(case):
    """About four times the error seen against `exact`; the iterative solves stop at their residual
    tolerance, which leaves more in the solution."""
    k = case["kind"]
    if k in ("apply", "force"):
        return dict(rel=3e-7 if case.get("f32") else 2e-14)
    if k == "explicit":
        return dict(rel=1e-5 if case["f32"] else 5e-14)
    if k == "static":
        return dict(rel=1e-7 if case["rtol"] > 1e-9 else 1e-9)
    if k in ("newmark", "j2"):
        return dict(rel=1e-10)
    if k in ("soil_force", "soil_stage", "points"):
        return dict(rel=1e-10)
    return dict(rel=1e-7)


# ---------------------------------------------------------------- the same in plain torch, 64 bits
class _Elements:
    """Gauss-point form of 8-node bricks: derivatives, volumes and materials of every element."""

    CORNERS = ((-1, -1, -1), (1, -1, -1), (1, 1, -1), (-1, 1, -1), (-1, -1, 1), (1, -1, 1), (1, 1, 1), (-1, 1, 1))

    def __init__(self, b):
        m = b.mesh
        E, P = m.count, m.padded
        self.n, self.m = m.num_equations, m
        eq = torch.as_tensor(m.eq.reshape(24, P)[:, :E].astype(np.int64), device=DEV)
        self.eq = torch.where(eq < 0, torch.full_like(eq, self.n), eq)
        node = torch.as_tensor(m.node.reshape(8, P)[:, :E].astype(np.int64), device=DEV)
        X = torch.as_tensor(m.coords.reshape(3, -1), device=DEV)[:, node]  # 3 8 E
        par = torch.as_tensor(m.params, device=DEV)[torch.as_tensor(m.param[:E].astype(np.int64), device=DEV)].T
        names = dict(zip(fx.PARAM_FIELDS, par))
        self.p = names
        self.mu = names["E"] / (2 * (1 + names["nu"]))
        self.lam = names["E"] * names["nu"] / ((1 + names["nu"]) * (1 - 2 * names["nu"]))
        self.points = []
        r = 1 / math.sqrt(3.0)
        for gp in range(8):
            g = [r if gp & s else -r for s in (4, 2, 1)]
            N = torch.tensor([np.prod([1 + c[d] * g[d] for d in range(3)]) / 8 for c in self.CORNERS], dtype=F64,
                             device=DEV)
            dn = torch.tensor([[c[d] * np.prod([1 + c[e] * g[e] for e in range(3) if e != d]) / 8
                                for c in self.CORNERS] for d in range(3)], dtype=F64, device=DEV)
            J = torch.einsum("dae,ka->edk", X, dn)
            dN = torch.einsum("ekd,ka->dae", torch.linalg.inv(J), dn).contiguous()
            self.points.append((N, dN, torch.linalg.det(J)))

    def gather(self, x):
        return torch.cat((x, x.new_zeros(1)))[self.eq].reshape(8, 3, -1)

    def scatter(self, ye):
        out = ye.new_zeros(self.n + 1)
        out.index_add_(0, self.eq.reshape(-1), ye.reshape(24, -1).reshape(-1))
        return out[:self.n]

    @staticmethod
    def strain(dN, ue):  # the symmetric gradient, 3 3 E
        G = torch.einsum("dae,ace->cde", dN, ue)
        return 0.5 * (G + G.transpose(0, 1))

    def stress(self, eps):
        s = 2 * self.mu * eps
        tr = self.lam * (eps[0, 0] + eps[1, 1] + eps[2, 2])
        for i in range(3):
            s[i, i] += tr
        return s

    def apply(self, x, k):
        """y = (k0 K + k1 C + k2 M) x with the elastic tangent."""
        p, xe = self.p, self.gather(x)
        ks = k[0] + k[1] * (p["betaK"] + p["betaKinit"] + p["betaKcomm"])
        cm = (k[2] + k[1] * p["alphaM"]) * p["rho"]
        lumped = p["mass_type"] == 1
        ye = torch.zeros_like(xe)
        for N, dN, det in self.points:
            s = self.stress(self.strain(dN, xe)) * (ks * det)
            ye += torch.einsum("dae,cde->ace", dN, s)
            v = torch.einsum("a,ace->ce", N, xe)
            ye += (cm * det) * N[:, None, None] * torch.where(lumped, xe, v[None])
        return self.scatter(ye)

    def body(self):
        ye = torch.zeros(8, 3, self.m.count, dtype=F64, device=DEV)
        b = torch.stack((self.p["b0"], self.p["b1"], self.p["b2"]))
        for N, _, det in self.points:
            ye += N[:, None, None] * (b * det)[None]
        return self.scatter(ye)

    def diagonal(self, k):
        p = self.p
        ks = k[0] + k[1] * (p["betaK"] + p["betaKinit"] + p["betaKcomm"])
        cm = (k[2] + k[1] * p["alphaM"]) * p["rho"]
        d = torch.zeros(8, 3, self.m.count, dtype=F64, device=DEV)
        for N, dN, det in self.points:
            sq = dN * dN
            full = self.mu * sq.sum(0)
            for c in range(3):
                d[:, c] += ks * det * (full + (self.lam + self.mu) * sq[c])
            n = N[:, None]
            d += (cm * det * torch.where(p["mass_type"] == 1, n, n * n))[:, None]
        return self.scatter(d)

    def solve(self, b, k, rtol):
        """Jacobi-PCG well past the tolerance of the path it checks."""
        inv = 1 / self.diagonal(k)
        x, r = torch.zeros_like(b), b.clone()
        z = inv * r
        p, rz, stop = z.clone(), torch.dot(r, z), rtol * b.norm()
        for it in range(20000):
            q = self.apply(p, k)
            a = rz / torch.dot(p, q)
            x += a * p
            r -= a * q
            if it % 8 == 7 and bool(r.norm() <= stop):
                break
            z = inv * r
            new = torch.dot(r, z)
            p = z + (new / rz) * p
            rz = new
        return x


def _j2_exact(b, f):
    """Newton on the radial return from the virgin state, dense tangents."""
    el = _Elements(b)
    p, n = el.p, el.n
    G, K = el.mu, p["E"] / (3 * (1 - 2 * p["nu"]))
    eye = torch.eye(3, dtype=F64, device=DEV)[:, :, None]
    u = torch.zeros(n, dtype=F64, device=DEV)
    first = None
    for _ in range(40):
        ue = el.gather(u)
        fe = torch.zeros_like(ue)
        A = torch.zeros(n + 1, n + 1, dtype=F64, device=DEV)
        keep = []
        for N, dN, det in el.points:
            eps = el.strain(dN, ue)
            tr = eps[0, 0] + eps[1, 1] + eps[2, 2]
            s = 2 * G * (eps - eye * tr / 3)
            norm = (s * s).sum((0, 1)).sqrt()
            over = norm - math.sqrt(2 / 3) * p["sigma_y"]
            dg = torch.clamp(over, min=0) / (2 * G + 2 / 3 * p["H"])
            nn = s / torch.where(norm > 0, norm, torch.ones_like(norm))
            sig = s - 2 * G * dg * nn + eye * (K * tr)
            theta = torch.where(over > 0, 1 - 2 * G * dg / torch.where(norm > 0, norm, torch.ones_like(norm)),
                                torch.ones_like(dg))
            bar = torch.where(over > 0, 1 / (1 + p["H"] / (3 * G)) - (1 - theta), torch.zeros_like(dg))
            fe += torch.einsum("dae,cde->ace", dN, sig * det)
            keep.append((dN, det, nn, theta, bar))
        r = f - el.scatter(fe)
        first = r.norm() if first is None else first
        if r.norm() <= 1e-12 * first:
            return u
        Ke = torch.zeros(el.m.count, 24, 24, dtype=F64, device=DEV)
        for dN, det, nn, theta, bar in keep:
            g2 = 2 * G * theta * det
            dot = torch.einsum("dae,dbe->abe", dN, dN)
            blk = torch.einsum("ae,be->abe", dN.reshape(24, -1), dN.reshape(24, -1)).reshape(3, 8, 3, 8, -1)
            # volumetric, deviatoric (symmetrised) and rank-one parts, indices (c a)(d b)
            k4 = blk.permute(1, 0, 3, 2, 4) * (K * det - g2 / 3) + 0.5 * g2 * blk.permute(1, 2, 3, 0, 4)
            k4 = k4 + 0.5 * g2 * dot[:, None, :, None] * torch.eye(3, dtype=F64, device=DEV)[None, :, None, :, None]
            w = torch.einsum("dae,cde->ace", dN, nn)
            k4 = k4 - (2 * G * bar * det) * w[:, :, None, None] * w[None, None]
            Ke += k4.reshape(24, 24, -1).permute(2, 0, 1)
        rows = el.eq.T[:, :, None].expand(-1, 24, 24)
        A.view(-1).index_add_(0, (rows * (n + 1) + el.eq.T[:, None, :]).reshape(-1), Ke.reshape(-1))
        u = u + torch.linalg.solve(A[:n, :n], r)
    return u


def exact(case, seed):
    k = case["kind"]
    if k in ("soil_force", "soil_stage", "points"):
        return None  # the multi-yield updates are path-dependent branches whose 64-bit form is the path's own
    if k == "apply" and case["mesh"] == "ssp":
        return None  # the stabilization's constants are a text of their own
    parts = _parts(case)
    b = parts[0]
    n = b.mesh.num_equations
    if k == "apply":
        x = _vector(seed, n)
        x = x.float().double() if case["f32"] else x
        return _Elements(b).apply(x, (1.0, case["damping"], case["mass"]))
    if k == "force":
        el, u, v = _Elements(b), _vector(seed, n, 1e-4), _vector(seed + 1, n, 1e-3)
        return el.apply(u, (1.0, 0.0, 0.0)) + el.apply(v, (0.0, 1.0, 0.0)) - el.body()
    if k == "explicit":
        el = _Elements(b)
        u, vh = _vector(seed, n, 1e-4), _vector(seed + 1, n, 1e-3)
        if case["f32"]:
            u, vh = u.float().double(), vh.float().double()
        dt = _explicit_dt(fx.InternalForce(b.mesh), case)
        mass = torch.as_tensor(b.mesh.lumped_mass, device=DEV)
        push = torch.as_tensor((b.dof == 0).astype(np.float64), device=DEV)
        a = torch.zeros_like(u)
        for g in _ground(seed, case["steps"], dt):
            vh = vh + dt * a
            u = u + dt * vh
            f = el.apply(u, (1.0, 0.0, 0.0)) + el.apply(vh, (0.0, 1.0, 0.0)) - el.body()
            new = -f / mass - push * float(g)
            v = vh + dt / 8 * (3 * new + a)
            a = new
        return u, vh, a, v
    if k == "static":
        return _Elements(b).solve(torch.as_tensor(_top_load(b, seed, 1e5), device=DEV), (1.0, 0.0, 0.0), 1e-14), 1.0
    if k == "newmark":
        el, dt = _Elements(b), NEWMARK_DT
        f, _ = stages.top_shear(b.spec, b.eqmap, 1e6)
        f = torch.as_tensor(f * np.random.default_rng(seed).uniform(0.5, 1.5, len(f)), device=DEV)
        u, v, a = (torch.zeros(n, dtype=F64, device=DEV) for _ in range(3))
        for i in range(case["steps"]):
            v, a = -v, -4 / dt * v - a
            r = f * math.sin(2 * math.pi * 5.0 * (i + 1) * dt) - el.apply(u, (1.0, 0.0, 0.0)) \
                - el.apply(v, (0.0, 1.0, 0.0)) - el.apply(a, (0.0, 0.0, 1.0))
            du = el.solve(r, (1.0, 2 / dt, 4 / dt ** 2), 1e-14)
            u, v, a = u + du, v + 2 / dt * du, a + 4 / dt ** 2 * du
        return [u, v, a]
    if k == "j2":
        out = []
        for i, part in enumerate(parts):
            u = _j2_exact(part, torch.as_tensor(_shear_load(part, seed + i, case["load"]), device=DEV))
            pad = (len(u) + 2047) // 2048 * 2048 if case["count"] > 1 else len(u)  # instances start at whole chunks
            out.append(torch.cat((u, u.new_zeros(pad - len(u)))))
        return torch.cat(out), 1.0
    return [_Elements(p).solve(torch.as_tensor(_top_load(p, seed + i, 1e5), device=DEV), (1.0, 0.0, 0.0), 1e-13)
            for i, p in enumerate(parts)]
