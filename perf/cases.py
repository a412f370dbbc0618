"""The work this framework does for its users, as measured cases.

A case is one whole job through the public Python API, as a caller writes it: the solver (or
batch) is created from host arrays, set up, stepped on the device, its fields are read back and
the handle is closed. Explicit dynamics has no call that can be repeated on an evolved handle
with the same answer, so the handle belongs to the pass; meshes, materials, defect fields and
the drawn parameters are what the caller already has and are made by ``prepare``.

The kinds:

* ``rod``    -- one Taylor rod on a rigid Coulomb anvil (scenes.taylor_rod), single scene;
* ``scene``  -- plane-strain bodies with penalty contact, friction, damage and erosion
                (scenes.perforation), single scene;
* ``tube``   -- the pressurised thin wall with damage at 2x2 points (scenes.tube);
* ``sweep``  -- a ragged batch of Taylor rods (scenes.sweep_instances) in one precision;
* ``burst``  -- a batch of tube wall slices with capacity sampling (scenes.burst_instance);
* ``adjoint``-- gradients of L/L0 of a batch of rods, forward with checkpoints and reverse;
* ``points`` -- the return map alone over arrays of material points.
"""
import math

import numpy as np

from neofiz_gb300 import (ExplicitSolver, Formulation, Integration, Kinematics, QuadMesh,
                          RigidWall, material_point_update)
from neofiz_gb300 import _abi, scenes
from neofiz_gb300.batch import BatchSolver

PRECISION = {"fp64": _abi.PRECISION_FP64, "mixed": _abi.PRECISION_MIXED,
             "compensated": _abi.PRECISION_COMPENSATED}
US = 1.0e-6
MM = 1.0e-3
RADIUS, LENGTH = 3.8e-3, 25.0e-3


def listed():
    return [
        # the smallest single scene of the tests: launches and the longest solve's chain count
        {"name": "rod-4x24", "kind": "rod", "nr": 4, "nz": 24, "steps": 400, "precision": "fp64"},
        # the 10 x 60 rod, the plain FP64 parity scene, over its first 1000 steps
        {"name": "rod-10x60", "kind": "rod", "nr": 10, "nz": 60, "steps": 1000,
         "precision": "fp64"},
        # a pressurised tube at 2x2 points with damage, to past the ramp's middle
        {"name": "tube-4x200", "kind": "tube", "nr": 4, "nz": 200, "steps": 600},
        # the 1 mm perforation: every contact, erosion and surface path on a small scene
        {"name": "perforation-1mm", "kind": "scene", "cell": 1.0, "steps": 400,
         "precision": "fp64"},
        # the headline scene, 200k quads, plain FP64, through the first of its impact
        {"name": "perforation-200k", "kind": "scene", "cell": 0.114, "steps": 300,
         "precision": "fp64"},
        # the 1M-quad scene in the mixed form
        {"name": "perforation-1M-mixed", "kind": "scene", "cell": 0.051, "steps": 400,
         "precision": "mixed"},
        # a parameter sweep that must equal its single scenes bit for bit
        {"name": "sweep-64-fp64", "kind": "sweep", "count": 64, "t_end": 4.0,
         "precision": "fp64"},
        # the same kind of sweep in the mixed form, more rods
        {"name": "sweep-256-mixed", "kind": "sweep", "count": 256, "t_end": 20.0,
         "precision": "mixed"},
        # the throughput form: half a thousand rods through the crush
        {"name": "sweep-512-comp", "kind": "sweep", "count": 512, "t_end": 30.0,
         "precision": "compensated"},
        # a burst sweep's many tiny instances, sampled as they run
        {"name": "burst-512", "kind": "burst", "count": 512, "steps": 3000, "precision": "fp64"},
        # design gradients of a batch of rods
        {"name": "adjoint-16", "kind": "adjoint", "count": 16, "nr": 10, "nz": 60,
         "t_end": 5.0},
        # the return map over a file of material points, host arrays in and out
        {"name": "points-60k", "kind": "points", "count": 60000},
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["rod", "rod", "scene", "scene", "tube", "sweep", "sweep", "burst",
                       "adjoint", "points"])
    if kind == "rod":
        nr = log(3, 60)
        return {"kind": kind, "nr": nr, "nz": nr * rng.randint(4, 7) + rng.randint(0, 3),
                "steps": rng.randint(150, 600), "precision": rng.choice(["fp64", "fp64", "mixed"])}
    if kind == "tube":
        return {"kind": kind, "nr": rng.randint(2, 7), "nz": log(11, 400),
                "steps": rng.randint(150, 500)}
    if kind == "scene":
        return {"kind": kind, "cell": round(math.exp(rng.uniform(math.log(0.09), 0.0)), 4),
                "steps": rng.randint(100, 280), "precision": rng.choice(["fp64", "mixed"])}
    if kind == "sweep":
        return {"kind": kind, "count": log(5, 300), "t_end": round(rng.uniform(2.0, 4.0), 2),
                "precision": rng.choice(["fp64", "mixed", "compensated"])}
    if kind == "burst":
        return {"kind": kind, "count": log(30, 900), "steps": rng.randint(500, 2500),
                "precision": rng.choice(["fp64", "compensated"])}
    if kind == "adjoint":
        nr = rng.randint(4, 11)
        return {"kind": kind, "count": log(2, 30), "nr": nr, "nz": rng.randint(4, 6) * nr + 1,
                "t_end": round(rng.uniform(2.0, 4.0), 2)}
    return {"kind": kind, "count": log(500, 150000)}


# ------------------------------------------------------------------------------ the inputs

def rods_of(case, seed):
    """Drawn rods in the sweep's ranges: Johnson-Cook A, B, n, C, friction and speed from the
    seed; a sweep's ragged meshes (nr 6..24, nz 30..120) from its size, so that every seed of a
    case has outputs of one shape."""
    g = np.random.RandomState(seed % (1 << 31))
    sizes = np.random.RandomState(case.get("count", 1))
    out = []
    for _ in range(case.get("count", 1)):
        nr, nz = int(sizes.randint(6, 25)), int(sizes.randint(30, 121))
        j = scenes.ROD_JC
        a, b, n, c = (v * g.uniform(0.8, 1.2) for v in (j.a, j.b, j.n, j.c))
        out.append({"nr": case.get("nr", nr), "nz": case.get("nz", nz), "a": a, "b": b, "n": n,
                    "c": c, "mu": g.uniform(0.0, 0.2), "speed": g.uniform(150.0, 250.0),
                    "t_end": case.get("t_end", 0.0) * US})
    return out


def points_of(case, seed):
    """Points of the rod steel on and off their yield surfaces, and one step's strains."""
    g = np.random.RandomState(seed % (1 << 31))
    n = case["count"]
    sig = g.uniform(-1.0, 1.0, (n, 4)) * 3.0e8
    back = g.uniform(-1.0, 1.0, (n, 4)) * 2.0e7
    back[:, :3] -= back[:, :3].mean(axis=1)[:, None]
    eps = np.where(g.uniform(size=n) < 0.4, 0.0, g.uniform(0.0, 0.4, n))
    work = eps * 5.0e8
    strain = g.uniform(-1.0, 1.0, (n, 4)) * 2.0e-3 * g.uniform(size=(n, 1))
    return {"sig": sig, "back": back, "eps": eps, "work": work, "strain": strain}


def prepare(case, seed):
    kind = case["kind"]
    state = {"case": dict(case)}
    if kind in ("rod", "sweep", "adjoint"):
        state["rods"] = rods_of(case, seed)
        state["instances"] = scenes.sweep_instances(state["rods"], RADIUS, LENGTH)
    elif kind == "scene":
        # the slug starts a hair from the blocks, so the steps are impact
        state["inputs"] = scenes.perforation_inputs(
            cell=case["cell"] * MM, speed=680.0 + seed % 41, seed=20240611 + seed % 100003,
            gap=0.02 * MM)
    elif kind == "tube":
        g = np.random.RandomState(seed % (1 << 31))
        nr, nz = case["nr"], case["nz"]
        mesh = QuadMesh.cylinderWall(19.6e-3, 20.4e-3, 0.8e-3 / nr * nz, nr, nz)
        state.update(mesh=mesh, ends=QuadMesh.axialEndNodes(nr, nz),
                     pressure=g.uniform(55.0e6, 65.0e6),
                     failure=scenes.tube_failure_strains(mesh, seed=1 + seed % 100003, scale=0.08))
    elif kind == "burst":
        g = np.random.RandomState(seed % (1 << 31))
        radii = g.uniform(10.0e-3, 40.0e-3, case["count"])
        slender = g.uniform(15.0, 60.0, case["count"])
        state["radii"] = radii
        state["instances"] = [scenes.burst_instance(float(r), float(s))
                              for r, s in zip(radii, slender)]
    else:
        state["points"] = points_of(case, seed)
        state["material"] = scenes.rod_material()
    return state


# ------------------------------------------------------------------------------ the passes

def _fields(s):
    return {"ur": s.radialDisplacement(), "uz": s.axialDisplacement(), "vr": s.velocityR(),
            "vz": s.velocityZ(), "stress": s.stress(), "plastic": s.plasticStrain(),
            "time": s.time()}


def _rod(state):
    case, inst, rod = state["case"], state["instances"][0], state["rods"][0]
    s = ExplicitSolver(inst.mesh, inst.material, Formulation.AXISYMMETRIC, Integration.REDUCED,
                       Kinematics.FINITE_STRAIN, 1.0, 0.6)
    s.setHourglassCoefficient(inst.hourglass)
    for n in inst.fixed_radial:
        s.fixRadial(n)
    s.setRigidWall(RigidWall.atZ(*inst.wall))
    s.setUniformVelocity(0.0, -rod["speed"])
    if case["precision"] == "mixed":
        s.setPrecision(PRECISION["mixed"])
    s.run(case["steps"])
    out = _fields(s)
    s.close()
    return out


def _scene(state):
    case = state["case"]
    s, _, _ = scenes.perforation_build(ExplicitSolver, state["inputs"])
    if case["precision"] == "mixed":
        s.setPrecision(PRECISION["mixed"])
    s.run(case["steps"])
    out = _fields(s)
    out["eroded"] = s.erodedElements()
    s.close()
    return out


def _tube(state):
    copper = scenes.tube_material()
    mesh = state["mesh"]
    s = ExplicitSolver(mesh, copper, Formulation.AXISYMMETRIC, Integration.FULL,
                       Kinematics.FINITE_STRAIN, 1.0, 0.5)
    for n in state["ends"]:
        s.fixAxial(n)
    s.setPressureRamp(state["pressure"], 10.0 * US)
    s.setRelaxationDamping(0.05, copper.barWaveSpeed() / 20.0e-3)
    s.setDamage(np.full(mesh.elementCount, scenes.TUBE_GF), state["failure"])
    s.run(state["case"]["steps"])
    out = _fields(s)
    s.close()
    return out


def _batch_fields(b):
    st, m = b.state(), b.measure()
    return {"ur": b.read(_abi.FIELD_UR), "uz": b.read(_abi.FIELD_UZ),
            "vr": b.read(_abi.FIELD_VR), "vz": b.read(_abi.FIELD_VZ),
            "stress": b.read(_abi.FIELD_STRESS), "plastic": b.read(_abi.FIELD_PLASTIC_STRAIN),
            "time": st["time"], "length": np.array([x.length for x in m]),
            "diameter": np.array([x.mushroom_diameter for x in m])}


def _sweep(state):
    b = BatchSolver(state["instances"], Formulation.AXISYMMETRIC, cfl=0.6,
                    precision=PRECISION[state["case"]["precision"]])
    b.run()
    out = _batch_fields(b)
    # the first rod by itself, as a caller plots one
    out["first"] = {"ur": b.readInstance(_abi.FIELD_UR, 0), "uz": b.readInstance(_abi.FIELD_UZ, 0),
                    "plastic": b.readInstance(_abi.FIELD_PLASTIC_STRAIN, 0)}
    b.close()
    return out


def _burst(state):
    case = state["case"]
    b = BatchSolver(state["instances"], Formulation.AXISYMMETRIC, cfl=scenes.BURST_CFL,
                    precision=PRECISION[case["precision"]])
    b.setBurst(scenes.BURST_SAMPLE_STEPS, state["radii"])
    b.run(case["steps"])
    out = _batch_fields(b)
    r = b.burstResults()
    out["capacity"], out["strain"], out["applied"] = r["capacity"], r["strain"], r["applied"]
    b.close()
    return out


def _adjoint(state):
    b = BatchSolver(state["instances"], Formulation.AXISYMMETRIC, cfl=0.6)
    b.adjointForward(200)
    values, grads = b.adjointBackward(_abi.OBJECTIVE_LENGTH_RATIO)
    b.close()
    return {"values": values, "grads": grads}


def _points(state):
    p = {k: v.copy() for k, v in state["points"].items()}
    dg = material_point_update(state["material"], p["sig"], p["back"], p["eps"], p["work"],
                               p["strain"], 2.0e-8, formulation=Formulation.AXISYMMETRIC)
    return {"sig": p["sig"], "back": p["back"], "eps": p["eps"], "work": p["work"],
            "multiplier": dg}


def run(state):
    return {"rod": _rod, "scene": _scene, "tube": _tube, "sweep": _sweep, "burst": _burst,
            "adjoint": _adjoint, "points": _points}[state["case"]["kind"]](state)


# ------------------------------------------------------------------------------ the work

def _rod_steps(nr, nz, t_end):
    """Steps of a rod to t_end (microseconds) at its first stable step."""
    edge = min(RADIUS / nr, LENGTH / nz)
    return t_end * US / (0.6 * edge / 5780.0) * 1.05


def work(case):
    """Bytes: each input once and each output once. Operations: FP64 (or FP32) operations of an
    elastic element-step (about 320 at one point, 1100 at 2x2; additions, multiplications,
    divisions and square roots each one), which every live element takes each step; return-map
    solves come on top and depend on the run. The reverse of a step is about three forwards."""
    kind = case["kind"]
    if kind == "points":
        return {"bytes": 8.0 * case["count"] * (14 + 11), "flops": 60.0 * case["count"]}
    points, per = 1, 320.0
    if kind == "rod":
        elements, steps, count = case["nr"] * case["nz"], case["steps"], 1
    elif kind == "tube":
        elements, steps, count, points, per = case["nr"] * case["nz"], case["steps"], 1, 4, 1100.0
    elif kind == "scene":
        elements, steps, count = int(2600.0 / case["cell"] ** 2), case["steps"], 1
    elif kind == "burst":
        elements, steps, count = 16, case["steps"], case["count"]
    elif kind == "adjoint":
        elements, count = case["nr"] * case["nz"], case["count"]
        steps, per = _rod_steps(case["nr"], case["nz"], case["t_end"]), 4 * 320.0
    else:
        elements, count = 1128, case["count"]
        steps = _rod_steps(14, 75, case["t_end"])
    # in: coordinates, connectivity, velocities; out: four nodal fields, stress, plastic strain
    return {"bytes": count * elements * (16.0 + 16.0 + 16.0 + 32.0 + points * 40.0),
            "flops": count * elements * steps * per}


# ------------------------------------------------------------------------------ in 64 bits

def _return_map(m, s, bk, eps, work, d, dt):
    """J2 return map with Johnson-Cook hardening over arrays of points, plain numpy."""
    lam = m["E"] * m["nu"] / ((1 + m["nu"]) * (1 - 2 * m["nu"]))
    mu = m["E"] / (2 * (1 + m["nu"]))
    k = m["k"]

    def thermal_term(w):
        h = k * w / (m["melt"] - m["room"])
        return np.where(h <= 0, 1.0, np.where(h >= 1, 0.0, 1.0 - np.clip(h, 1e-300, 1.0) ** m["m"]))

    def strain_term(e):
        return np.where(e > 0, m["a"] + m["b"] * np.maximum(e, 1e-300) ** m["n"], m["a"])

    r23 = math.sqrt(2.0 / 3.0)
    trial = s + 2 * mu * np.stack([d[:, 0], d[:, 1], d[:, 2], 0.5 * d[:, 3]], axis=1)
    trial[:, :3] += (lam * d[:, :3].sum(axis=1))[:, None]
    x = trial - bk
    x[:, :3] -= (trial[:, :3].sum(axis=1) / 3.0)[:, None]
    norm = np.sqrt((x[:, :3] ** 2).sum(axis=1) + 2 * x[:, 3] ** 2)
    th = thermal_term(work)
    plastic = np.nonzero(norm > r23 * strain_term(eps) * th)[0]
    dg = np.zeros(len(eps))
    s[:] = trial
    if plastic.size:
        nm, e0, t0 = norm[plastic], eps[plastic], th[plastic]
        stiff = 2 * mu + 2.0 / 3.0 * m["kin"]
        lo, hi = np.zeros(len(nm)), nm / stiff
        g = hi.copy()
        live = np.arange(len(nm))
        for _ in range(25):
            if not live.size:
                break
            gl, el, tl, nl = g[live], e0[live], t0[live], nm[live]
            e = el + r23 * gl
            rate = r23 * gl / dt
            st = strain_term(e)
            fast = rate > m["ref"]
            rf = np.where(fast, 1 + m["c"] * np.log(np.maximum(rate / m["ref"], 1e-300)), 1.0)
            f = nl - stiff * gl - r23 * st * rf * tl
            up = f > 0
            lo[live] = np.where(up, gl, lo[live])
            hi[live] = np.where(up, hi[live], gl)
            go = np.abs(f) > 1e-10 * m["a"]
            slope = -stiff - 2.0 / 3.0 * (m["n"] * (st - m["a"]) / e) * rf * tl
            slope = np.where(fast, slope - r23 * st * m["c"] * tl / gl, slope)
            new = gl - f / slope
            a, b = lo[live], hi[live]
            new = np.where((new > a) & (new < b), new, 0.5 * (a + b))
            g[live[go]] = new[go]
            live = live[go]
        n = x[plastic] / nm[:, None]
        pull = 2 * mu * g
        alpha = (bk[plastic][:, :3] * n[:, :3]).sum(axis=1) + 2 * bk[plastic][:, 3] * n[:, 3]
        s[plastic] -= pull[:, None] * n
        work[plastic] += g * (nm - pull + alpha)
        bk[plastic] += (2.0 / 3.0 * m["kin"] * g)[:, None] * n
        eps[plastic] += r23 * g
        dg[plastic] = g
    return dg


def _steel(rod):
    """The rod steel's constants with a drawn Johnson-Cook law (kinematic modulus 0.3 of the
    law's secant at 0.6 strain)."""
    return {"E": 200.0e9, "nu": 0.29, "rho": 7850.0, "a": rod["a"], "b": rod["b"], "n": rod["n"],
            "c": rod["c"], "m": 1.0, "ref": 1.0, "room": 293.0, "melt": 1793.0,
            "k": 0.9 / (7850.0 * 477.0), "kin": 0.3 * rod["b"] * 0.6 ** rod["n"] / 0.6}


def _rod_exact(rod, steps=None):
    """A Taylor rod stepped in numpy: one-point quads, Cayley co-rotation, hourglass stiffness
    0.10, a Coulomb wall at z = 0, the adaptive step; `steps` steps, or while time < t_end."""
    m, nr, nz = _steel(rod), rod["nr"], rod["nz"]
    i, j = np.arange(nr + 1.0), np.arange(nz + 1.0)
    X = np.stack([np.tile(RADIUS * i / nr, nz + 1), np.repeat(LENGTH * j / nz, nr + 1)], axis=1)
    base = (np.arange(nz)[:, None] * (nr + 1) + np.arange(nr)[None, :]).reshape(-1)
    c = np.stack([base, base + 1, base + nr + 2, base + nr + 1], axis=1)
    N, E = len(X), len(c)
    mu = m["E"] / (2 * (1 + m["nu"]))
    lam = m["E"] * m["nu"] / ((1 + m["nu"]) * (1 - 2 * m["nu"]))
    wave = math.sqrt((lam + 2 * mu) / m["rho"])
    mass = np.zeros(N)
    G = 1 / math.sqrt(3.0)
    p = X[c]
    for xi, eta in ((-G, -G), (G, -G), (G, G), (-G, G)):
        sh = 0.25 * np.array([(1 - xi) * (1 - eta), (1 + xi) * (1 - eta), (1 + xi) * (1 + eta),
                              (1 - xi) * (1 + eta)])
        dx = 0.25 * np.array([-(1 - eta), 1 - eta, 1 + eta, -(1 + eta)])
        de = 0.25 * np.array([-(1 - xi), -(1 + xi), 1 + xi, 1 - xi])
        jx, je = np.einsum("k,ekd->ed", dx, p), np.einsum("k,ekd->ed", de, p)
        vol = 2 * np.pi * (p[:, :, 0] @ sh) * (jx[:, 0] * je[:, 1] - jx[:, 1] * je[:, 0])
        np.add.at(mass, c.reshape(-1), (m["rho"] * vol[:, None] * sh[None, :]).reshape(-1))
    axis = np.arange(nz + 1) * (nr + 1)
    U, V, F = np.zeros((N, 2)), np.zeros((N, 2)), np.zeros((N, 2))
    V[:, 1] = -rod["speed"]
    s, bk, hg = np.zeros((E, 4)), np.zeros((E, 4)), np.zeros((E, 2))
    eps, wp = np.zeros(E), np.zeros(E)
    on = np.zeros(N, bool)
    edge = min(float(np.min(np.hypot(*(p[:, k] - p[:, (k + 1) % 4]).T))) for k in range(4))
    dt = old = 0.6 * edge / wave
    time, fixed = 0.0, np.zeros(N, bool)
    fixed[axis] = True
    sign = np.array([1.0, -1.0, 1.0, -1.0])
    flat = c.reshape(-1)
    taken = 0
    while (taken < steps) if steps is not None else (time < rod["t_end"]):
        avg = 0.5 * (old + dt)
        rest = on & (F[:, 1] <= 0)
        free = V[:, 0] + avg * F[:, 0] / mass
        if rod["mu"] > 0:
            tr = -mass * V[:, 0] / avg - F[:, 0]
            lim = rod["mu"] * -F[:, 1]
            slid = V[:, 0] + avg * (F[:, 0] + np.copysign(lim, tr)) / mass
            free = np.where(rest, np.where(np.abs(tr) <= lim, 0.0, slid), free)
        V[:, 0] = np.where(fixed, 0.0, free)
        U[:, 0] += V[:, 0] * dt
        vz = V[:, 1] + avg * F[:, 1] / mass
        z = X[:, 1] + U[:, 1]
        arrive = ~rest & (z + vz * dt < 0.0)
        go = ~rest & ~arrive
        U[:, 1] = np.where(arrive, U[:, 1] - z, np.where(go, U[:, 1] + vz * dt, U[:, 1]))
        V[:, 1] = np.where(arrive, 0.0, np.where(go, vz, V[:, 1]))
        on = rest | arrive
        time += dt
        taken += 1
        q = (X + U - 0.5 * dt * V)[c]
        dv = V[c] * dt
        short = min(float(np.min(((q[:, k] - q[:, (k + 1) % 4]) ** 2).sum(axis=1)))
                    for k in range(4))
        r, zz = q[:, :, 0], q[:, :, 1]
        gx, ge = 0.25 * np.array([-1, 1, 1, -1.0]), 0.25 * np.array([-1, -1, 1, 1.0])
        J00, J01, J10, J11 = r @ gx, zz @ gx, r @ ge, zz @ ge
        det = J00 * J11 - J01 * J10
        dr = (np.outer(J11, gx) - np.outer(J01, ge)) / det[:, None]
        dz = (-np.outer(J10, gx) + np.outer(J00, ge)) / det[:, None]
        a, b = dv[:, :, 0], dv[:, :, 1]
        rg = r.mean(axis=1)
        rz, zr = (dz * a).sum(axis=1), (dr * b).sum(axis=1)
        d = np.stack([(dr * a).sum(axis=1), (dz * b).sum(axis=1), a.mean(axis=1) / rg, rz + zr],
                     axis=1)
        h = 0.25 * (zr - rz)
        cs, sn = (1 - h * h) / (1 + h * h), 2 * h / (1 + h * h)
        for t in (s, bk):
            t0, t1, t3 = t[:, 0].copy(), t[:, 1].copy(), t[:, 3].copy()
            t[:, 0] = cs * cs * t0 - 2 * cs * sn * t3 + sn * sn * t1
            t[:, 1] = sn * sn * t0 + 2 * cs * sn * t3 + cs * cs * t1
            t[:, 3] = cs * sn * (t0 - t1) + (cs * cs - sn * sn) * t3
        _return_map(m, s, bk, eps, wp, d, dt)
        vol = 4 * 2 * np.pi * rg * det
        f = np.empty((E, 4, 2))
        f[:, :, 0] = -((dr * s[:, 0:1] + dz * s[:, 3:4]) * vol[:, None]
                       + (0.25 * s[:, 2] / rg * vol)[:, None])
        f[:, :, 1] = -(dz * s[:, 1:2] + dr * s[:, 3:4]) * vol[:, None]
        hr, hz = r @ sign, zz @ sign
        y = sign[None, :] - hr[:, None] * dr - hz[:, None] * dz
        kk = 0.10 * mu * vol * ((dr ** 2).sum(axis=1) + (dz ** 2).sum(axis=1))
        hg[:, 0] += kk * (y * a).sum(axis=1)
        hg[:, 1] += kk * (y * b).sum(axis=1)
        f -= y[:, :, None] * hg[:, None, :]
        F = np.stack([np.bincount(flat, f[:, :, k].reshape(-1), N) for k in (0, 1)], axis=1)
        old, dt = dt, 0.6 * math.sqrt(short) / wave
    return U, V, s, eps, time


def exact(case, seed):
    kind = case["kind"]
    if kind == "points":
        p = points_of(case, seed)
        rod = {"a": 350.0e6, "b": 275.0e6, "n": 0.36, "c": 0.022}
        dg = _return_map(_steel(rod), p["sig"], p["back"], p["eps"], p["work"], p["strain"],
                         2.0e-8)
        return {"sig": p["sig"], "back": p["back"], "eps": p["eps"], "work": p["work"],
                "multiplier": dg}
    if kind == "rod" and case["nr"] * case["nz"] * case["steps"] < 2.0e6:
        U, V, s, eps, time = _rod_exact(rods_of(case, seed)[0], case["steps"])
        return {"ur": U[:, 0], "uz": U[:, 1], "vr": V[:, 0], "vz": V[:, 1],
                "stress": s.reshape(-1), "plastic": eps, "time": time}
    if kind == "sweep":
        U, _, _, eps, _ = _rod_exact(rods_of(case, seed)[0])
        return {"ur": None, "uz": None, "vr": None, "vz": None, "stress": None, "plastic": None,
                "time": None, "length": None, "diameter": None,
                "first": {"ur": U[:, 0], "uz": U[:, 1], "plastic": eps}}
    return None
