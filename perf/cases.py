"""Performance cases of moleculardynamics_b200: what its users have it do, each through
the package's public entry points, from host state to host state.

Every case builds its own inputs from a seed (a jittered fcc lattice of Lennard-Jones
atoms or a lattice of randomly turned rigid SPC/E molecules, with Maxwell-Boltzmann
velocities), keeps the handles a program keeps (system, list, force field, integrator,
pinned host columns) and runs one pass: a force call, a stretch of a trajectory, a
batch, a gradient.  exact() is the same mathematics in plain 64-bit torch.
"""
import ctypes as C
import math

import numpy as np
import torch

import moleculardynamics_b200 as md

F64 = torch.float64
DT = 0.005                     # LJ time step
TAU_PS = 1.0966875353          # the water time unit in ps
O_SIGMA, O_EPS, Q_H = 3.16555789, 78.19743111, 0.42380
M_O, M_H = 15.9994, 1.008
R_OH, ANGLE = 1.0, 109.47


def listed():
    return [
        # One step of the drop-in loop, step(System&, ForceFn): the smallest call, where
        # launches and the round trips to the host are all there is.
        dict(name="lj_step_500", kind="step", nx=5, ny=5, nz=5, density=0.8442, rc=2.5, skin=0.3,
             steps=1, shift=False, precision="fp64"),
        # The 864-atom argon-like fluid, moldyn_run's own size, in the fused loop with a
        # thermo row per step.
        dict(name="lj_nve_864_fp64", kind="run", nx=6, ny=6, nz=6, density=0.8442, rc=2.5, skin=0.3,
             steps=50, shift=False, precision="fp64", integrator="vv"),
        # The large liquid in both precisions (the headline workload).
        dict(name="lj_nve_1m_mixed", kind="run", nx=64, ny=64, nz=64, density=0.8442, rc=2.5,
             skin=0.3, steps=40, shift=False, precision="mixed", integrator="vv"),
        dict(name="lj_nve_1m_fp64", kind="run", nx=64, ny=64, nz=64, density=0.8442, rc=2.5,
             skin=0.3, steps=40, shift=False, precision="fp64", integrator="vv"),
        # Langevin equilibration of a mid-sized system, odd in every direction.
        dict(name="lj_langevin_117k_mixed", kind="run", nx=31, ny=29, nz=31, density=0.8442, rc=2.5,
             skin=0.3, steps=40, shift=False, precision="mixed", integrator="baoab"),
        # Energy and forces of one configuration from host arrays: list build and force
        # pass of a moderately dense fluid in an oblong box, vacancies included.
        dict(name="lj_config_oblong_fp64", kind="config", nx=53, ny=37, nz=29, density=0.5, rc=3.0,
             skin=0.3, missing=1013, shift=True, precision="fp64", source="verlet"),
        # A sweep of independent Nose-Hoover replicas, 256 to 32,000 atoms, gas to liquid.
        dict(name="lj_batch_48_mixed", kind="batch", replicas=48, small=4, large=20, table=20261203,
             steps=40, precision="mixed"),
        # Rigid water with PME, SETTLE and FP32 real-space terms, thermostatted.
        dict(name="water_4096_pme_mixed", kind="water", per_side=16, rc=10.0, alpha=0.34, kmax=0,
             spacing=0.8, precision="mixed", settle=True, thermostat=True, steps=40),
        # Energy and forces of the same box from the k-vector sums, all FP64.
        dict(name="water_4096_ewald_fp64", kind="spce", per_side=16, rc=10.0, alpha=0.34, kmax=18,
             precision="fp64"),
        # The small water box of the water_rdf protocol: SHAKE/RATTLE, k-vector sums, a
        # velocity rescale after every 50 steps.
        dict(name="water_343_shake_fp64", kind="water", per_side=7, rc=10.0, alpha=0.0, kmax=5,
             spacing=0.0, precision="fp64", settle=False, thermostat=False, steps=50),
        # Loss gradient of a differentiable trajectory (forward and backward).
        dict(name="lj_adjoint_32000", kind="adjoint", cells=20, density=0.8442, steps=50, every=25,
             skin=1.0),
        # Production analysis: g(r), MSD and VACF frames taken along an FP64 trajectory.
        dict(name="lj_analysis_108k", kind="analysis", cells=30, density=0.8442, frames=4, stride=5,
             rmax=4.0, bins=200, max_lag=100),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "run", "run", "run", "config", "batch", "water", "water", "spce",
                       "adjoint", "analysis"])
    precision = rng.choice(["fp64", "mixed"])
    density = rng.choice([0.1, 0.3, 0.5, 0.7, 0.8, 0.8442])
    if kind in ("step", "run", "config"):
        side = math.exp(rng.uniform(math.log(4.0), math.log({"step": 20, "run": 60, "config": 52}[kind])))
        n = [max(4, int(round(side * rng.uniform(0.85, 1.07)))) for _ in range(3)]
        case = dict(kind=kind, nx=n[0], ny=n[1], nz=n[2], density=density, rc=2.5, skin=0.3,
                    shift=rng.random() < 0.4, precision=precision)
        if kind == "step":
            case.update(steps=rng.randint(1, 4), precision="fp64")
        elif kind == "run":
            integrator = rng.choice(["vv", "vv", "nhc", "baoab"])
            if precision == "mixed" and integrator != "baoab":
                case["shift"] = rng.random() < 0.8
            case.update(steps=rng.randint(10, 40), integrator=integrator)
            if precision == "mixed":  # the fixed-point path of a cubic and of an oblong box
                if rng.random() < 0.7:
                    case.update(ny=n[0], nz=n[0])
        else:
            case.update(missing=rng.randint(0, n[0] * n[1]), source=rng.choice(["verlet", "verlet", "cells"]),
                        rc=rng.choice([2.5, 3.0]), precision="fp64" if rng.random() < 0.7 else "mixed")
            if case["source"] == "cells":
                case["precision"] = "fp64"
        return case
    if kind == "batch":
        return dict(kind=kind, replicas=_log_int(rng, 4, 48), small=4, large=rng.randint(6, 20),
                    table=rng.randint(1, 1 << 20), steps=rng.randint(10, 40), precision=precision)
    if kind == "water":
        pme = rng.random() < 0.6
        per_side = rng.randint(8, 16) if pme else rng.randint(7, 8)
        return dict(kind=kind, per_side=per_side, rc=rng.choice([9.0, 10.0]) if per_side > 7 else 9.0,
                    alpha=0.34 if pme else 0.0, kmax=0 if pme else rng.randint(5, 7),
                    spacing=rng.choice([0.8, 0.9, 1.0]) if pme else 0.0, precision=precision,
                    settle=rng.random() < 0.5, thermostat=rng.random() < 0.5, steps=rng.randint(10, 40))
    if kind == "spce":
        per_side = rng.randint(7, 16)
        return dict(kind=kind, per_side=per_side, rc=9.0 if per_side < 8 else 10.0, alpha=0.34,
                    kmax=max(5, int(per_side * rng.uniform(0.9, 1.12))), precision=precision)
    if kind == "adjoint":
        steps = rng.randint(10, 50)
        return dict(kind=kind, cells=rng.randint(5, 20), density=0.8442, steps=steps,
                    every=rng.randint(5, max(5, steps // 2)), skin=1.0)
    return dict(kind=kind, cells=rng.randint(8, 30), density=rng.choice([0.5, 0.7, 0.8442]),
                frames=rng.randint(2, 4), stride=rng.randint(1, 5), rmax=4.0,
                bins=rng.choice([100, 200, 300]), max_lag=rng.randint(20, 100))


# --------------------------------------------------------------------------- inputs
def _generator(seed):
    g = torch.Generator()
    g.manual_seed(int(seed) & 0x7FFFFFFF)
    return g


def _lattice(nx, ny, nz, density, temperature, g, missing=0):
    """fcc lattice of nx x ny x nz cells in the box [-L/2, L/2), each atom moved by up to
    0.1 per axis, unit masses, velocities at `temperature` without centre-of-mass motion."""
    a = (4.0 / density) ** (1.0 / 3.0)
    basis = torch.tensor([[0.0, 0, 0], [0.5, 0.5, 0], [0.5, 0, 0.5], [0, 0.5, 0.5]], dtype=F64)
    cell = torch.cartesian_prod(*[torch.arange(k, dtype=F64) for k in (nx, ny, nz)])
    box = torch.tensor([nx * a, ny * a, nz * a], dtype=F64)
    pos = ((cell[:, None, :] + basis + 0.25) * a).reshape(-1, 3)
    if missing:
        keep = torch.randperm(len(pos), generator=g)[missing:].sort().values
        pos = pos[keep]
    pos = pos - 0.5 * box + 0.2 * (torch.rand(pos.shape, generator=g, dtype=F64) - 0.5)
    pos = pos - box * torch.floor(pos / box + 0.5)
    vel = math.sqrt(temperature) * torch.randn(pos.shape, generator=g, dtype=F64)
    return pos.numpy(), (vel - vel.mean(0)).numpy(), box.numpy()


def _water(per_side, g):
    """per_side^3 randomly turned SPC/E molecules at 0.997 g/cm^3 in O, H, H order, and
    298 K velocities that respect the bonds (rigid translation and rotation)."""
    m = per_side ** 3
    box = per_side * (18.01528 / 6.02214076e23 / 0.997 * 1e24) ** (1.0 / 3.0)
    half = 0.5 * math.radians(ANGLE)
    local = torch.tensor([[0.0, 0, 0], [R_OH * math.sin(half), 0, R_OH * math.cos(half)],
                          [-R_OH * math.sin(half), 0, R_OH * math.cos(half)]], dtype=F64)
    q, _ = torch.linalg.qr(torch.randn((m, 3, 3), generator=g, dtype=F64))
    centre = (torch.cartesian_prod(*[torch.arange(per_side, dtype=F64)] * 3) + 0.5) * (box / per_side)
    body = torch.einsum("mij,kj->mki", q, local)
    pos = (centre[:, None, :] + body).reshape(-1, 3) - 0.5 * box
    mass = torch.tensor([M_O, M_H, M_H], dtype=F64)
    com = (body * mass[:, None]).sum(1, keepdim=True) / mass.sum()
    omega = 0.05 * math.sqrt(298.0) * torch.randn((m, 1, 3), generator=g, dtype=F64)
    vcom = math.sqrt(298.0 / float(mass.sum())) * torch.randn((m, 1, 3), generator=g, dtype=F64)
    vel = (vcom - vcom.mean(0) + torch.linalg.cross(omega.expand(m, 3, 3), body - com)).reshape(-1, 3)
    return pos.numpy(), vel.numpy(), np.full(3, box), mass.repeat(m).numpy()


def _charges(m):
    return np.tile([-2.0 * Q_H, Q_H, Q_H], m)


def _lj_of(case):
    return md.LennardJones(1.0, 1.0, case.get("rc", 2.5),
                           md.Truncation.LinearForceShift if case.get("shift") else md.Truncation.Truncated,
                           precision=_precision(case))


def _precision(case):
    return md.PRECISION_MIXED if case["precision"] == "mixed" else md.PRECISION_FP64


def _table(case, seed):
    """The batch's replicas (cells, density, temperature): fixed by the case, as a sweep's
    plan is; the seed moves their atoms."""
    t = np.random.default_rng(case["table"])
    rows = []
    for k in range(case["replicas"]):
        cells = int(t.integers(case["small"], case["large"] + 1))
        rho = float([0.1, 0.3, 0.5, 0.7, 0.8, 0.9][int(t.integers(0, 6))])
        temp = float(t.uniform(1.0, 2.0))
        pos, vel, box = _lattice(cells, cells, cells, rho, temp, _generator(seed * 1009 + k))
        rows.append((pos, vel, box, temp))
    return rows


class _Columns:
    """Pinned host columns of some fields of a system, filled by one library call."""

    def __init__(self, n, fields):
        self.host = torch.empty((len(fields), n), dtype=F64, pin_memory=True)
        self.fields = (C.c_int * len(fields))(*fields)
        self.ptrs = (C.POINTER(C.c_double) * len(fields))(
            *[C.cast(row.data_ptr(), C.POINTER(C.c_double)) for row in self.host])

    def read(self, sys):
        md._check(md.lib().md_system_get_fields(sys.handle, len(self.fields), self.fields, self.ptrs))
        return self.host

    def write(self, sys):
        md._check(md.lib().md_system_set_fields(sys.handle, len(self.fields), self.fields, self.ptrs))


STATE = (md.FIELD_X, md.FIELD_Y, md.FIELD_Z, md.FIELD_VX, md.FIELD_VY, md.FIELD_VZ)
PLACE = STATE[:3]
FORCE = (md.FIELD_FX, md.FIELD_FY, md.FIELD_FZ)


def _steps_tau(fs):
    return fs * 1e-3 / TAU_PS


def _lj_inputs(case, seed):
    temp = 0.722 if case["density"] > 0.6 else 1.5
    return _lattice(case["nx"], case["ny"], case["nz"], case["density"], temp, _generator(seed),
                    case.get("missing", 0)) + (temp,)


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind in ("step", "run"):
        pos, vel, box, temp = _lj_inputs(case, seed)
        n = len(pos)
        s["sys"] = md.System.from_arrays(pos, box, vel=vel, mass=np.ones(n))
        s["lj"] = _lj_of(case)
        s["list"] = md.VerletList(box, case["rc"], case["skin"])
        s["list"].build(s["sys"])
        s["lj"].compute_forces(s["sys"], s["list"])
        which = case.get("integrator", "vv")
        s["it"] = (md.VelocityVerlet(DT) if which == "vv" else
                   md.NoseHooverChain(DT, temp, 0.5, 3, 3 * n - 3) if which == "nhc" else
                   md.LangevinBAOAB(DT, 1.0, temp, seed & 0xFFFF))
        s["out"] = _Columns(n, STATE + (FORCE if kind == "step" else ()))
    elif kind == "config":
        pos, vel, box, _ = _lj_inputs(case, seed)
        n = len(pos)
        s["sys"] = md.System.from_arrays(pos, box, mass=np.ones(n))
        s["lj"] = _lj_of(case)
        s["list"] = (md.CellList(box, case["rc"]) if case["source"] == "cells" else
                     md.VerletList(box, case["rc"], case["skin"]))
        s["in"], s["out"] = _Columns(n, PLACE), _Columns(n, FORCE)
        s["in"].host.copy_(torch.from_numpy(pos.T.copy()))
    elif kind == "batch":
        s["batch"], s["parts"] = md.Batch(), []
        rows = _table(case, seed)
        total, at = sum(len(r[0]) for r in rows), 0
        s["host"] = torch.empty((6, total), dtype=F64, pin_memory=True)
        for pos, vel, box, temp in rows:
            n = len(pos)
            ctx = md.Context(0)
            sys = md.System.from_arrays(pos, box, vel=vel, mass=np.ones(n), ctx=ctx)
            lj = md.LennardJones(1.0, 1.0, 2.5, precision=_precision(case))
            v = md.VerletList(box, 2.5, 0.3, ctx=ctx)
            v.build(sys)
            lj.compute_forces(sys, v)
            s["batch"].add(md.NoseHooverChain(DT, temp, 0.5, 3, 3 * n - 3), sys, v, lj)
            ptrs = (C.POINTER(C.c_double) * 6)(
                *[C.cast(row[at:].data_ptr(), C.POINTER(C.c_double)) for row in s["host"]])
            s["parts"].append((sys, ptrs))
            at += n
        s["fields"] = (C.c_int * 6)(*STATE)
    elif kind in ("water", "spce"):
        pos, vel, box, mass = _water(case["per_side"], _generator(seed))
        m = len(pos) // 3
        s["sys"] = md.System.from_arrays(pos, box, vel=vel, mass=mass, charge=_charges(m),
                                         mol=np.arange(3 * m) // 3)
        s["ff"] = md.SpceForceField(cutoff=case["rc"], kmax=case["kmax"], alpha=case["alpha"])
        s["ff"].set_precision(_precision(case))
        if kind == "spce":
            s["in"], s["out"] = _Columns(3 * m, PLACE), _Columns(3 * m, FORCE)
            s["in"].host.copy_(torch.from_numpy(pos.T.copy()))
        else:
            if case["spacing"] > 0:
                s["ff"].set_pme_spacing(box, case["spacing"], 6)
            rigid = md.RigidWater(R_OH, ANGLE, settle=case["settle"])
            s["dof"] = md.RigidWater.degrees_of_freedom(m, True)
            dt = _steps_tau(1.0)
            s["it"] = (md.ConstrainedNoseHooverChain(dt, rigid, 298.0, _steps_tau(100.0), 3, s["dof"])
                       if case["thermostat"] else md.ConstrainedVelocityVerlet(dt, rigid))
            s["out"] = _Columns(3 * m, STATE)
    elif kind == "adjoint":
        c = case["cells"]
        pos, vel, box = _lattice(c, c, c, case["density"], 0.722, _generator(seed))
        s["sys"] = md.System.from_arrays(pos, box, vel=vel, mass=np.ones(len(pos)))
        s["in"] = _Columns(len(pos), STATE)
        s["in"].host.copy_(torch.from_numpy(np.concatenate([pos.T, vel.T])))
        s["lj"] = md.LennardJones(1.0, 1.0, 2.5, md.Truncation.LinearForceShift)
        s["traj"] = md.AdjointTrajectory()
        s["grad"] = _adjoint_weights(case, len(pos), seed)
    else:
        c = case["cells"]
        pos, vel, box = _lattice(c, c, c, case["density"], 0.722, _generator(seed))
        n = len(pos)
        s["sys"] = md.System.from_arrays(pos, box, vel=vel, mass=np.ones(n))
        s["lj"] = md.LennardJones(1.0, 1.0, 2.5)
        s["list"] = md.VerletList(box, 2.5, 0.3)
        s["list"].build(s["sys"])
        s["lj"].compute_forces(s["sys"], s["list"])
        s["it"] = md.VelocityVerlet(DT)
        s["rdf"] = md.Rdf(case["rmax"], case["bins"])
        s["msd"], s["vacf"] = md.Msd(n, case["max_lag"]), md.Vacf(n, case["max_lag"])
        s["out"] = _Columns(n, STATE)
    return s


def _adjoint_weights(case, n, seed):
    """dL/d(U, W, KE) of a loss on the time-averaged energy and pressure."""
    w = torch.rand((case["steps"], 3), generator=_generator(seed + 77), dtype=F64).numpy()
    return (0.5 + w) / (n * case["steps"])


# ------------------------------------------------------------------------- one pass
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "step":
        def force_fn(sys):
            s["list"].rebuild_if_needed(sys)
            return s["lj"].compute_forces(sys, s["list"])
        for _ in range(case["steps"]):
            e, w = s["it"].step(s["sys"], force_fn)
        h = s["out"].read(s["sys"])
        return {"energy": np.float64(e), "virial": np.float64(w), "pos": h[:3], "vel": h[3:6],
                "force": h[6:]}
    if kind == "run":
        rows = s["it"].run(s["sys"], s["list"], s["lj"], case["steps"], thermo=True)
        h = s["out"].read(s["sys"])
        return {"energy": rows[:, 0], "virial": rows[:, 1], "kinetic": rows[:, 2],
                "conserved": rows[:, 3], "pos": h[:3], "vel": h[3:]}
    if kind == "config":
        s["in"].write(s["sys"])
        s["list"].build(s["sys"])
        e, w = s["lj"].compute_forces(s["sys"], s["list"])
        return {"energy": np.float64(e), "virial": np.float64(w), "force": s["out"].read(s["sys"])}
    if kind == "batch":
        rows = s["batch"].run(case["steps"], thermo=True)
        lib = md.lib()
        for sys, ptrs in s["parts"]:
            md._check(lib.md_system_get_fields(sys.handle, 6, s["fields"], ptrs))
        return {"energy": rows[:, :, 0], "virial": rows[:, :, 1], "kinetic": rows[:, :, 2],
                "conserved": rows[:, :, 3], "pos": s["host"][:3], "vel": s["host"][3:]}
    if kind == "spce":
        s["in"].write(s["sys"])
        e = s["ff"].compute_forces(s["sys"])
        return {"energy": np.float64(e), "virial": np.float64(s["ff"].parts["virial"]),
                "force": s["out"].read(s["sys"])}
    if kind == "water":
        rows = s["it"].run(s["sys"], s["ff"], case["steps"], thermo=True)
        if not case["thermostat"]:
            s["sys"].rescale_temperature(s["dof"], 298.0)
        h = s["out"].read(s["sys"])
        return {"energy": rows[:, 0], "virial": rows[:, 1], "kinetic": rows[:, 2],
                "conserved": rows[:, 3], "pos": h[:3], "vel": h[3:]}
    if kind == "adjoint":
        s["in"].write(s["sys"])
        rows = s["traj"].forward(s["sys"], s["lj"], DT, case["steps"], case["every"], case["skin"])
        de, ds, gx, gv = s["traj"].backward(s["grad"])
        return {"rows": rows, "d_epsilon": np.float64(de), "d_sigma": np.float64(ds), "d_pos": gx,
                "d_vel": gv}
    for _ in range(case["frames"]):
        s["it"].run(s["sys"], s["list"], s["lj"], case["stride"])
        s["rdf"].accumulate(s["sys"])
        s["msd"].push(s["sys"])
        s["vacf"].push(s["sys"])
    h = s["out"].read(s["sys"])
    return {"histogram": s["rdf"].histogram().astype(np.int64), "g": s["rdf"].g(),
            "msd": s["msd"].msd(), "vacf": s["vacf"].vacf(), "pos": h[:3], "vel": h[3:]}


# ----------------------------------------------------------------- what it cannot avoid
def _pairs_per_atom(density, r):
    return 0.5 * 4.0 / 3.0 * math.pi * r ** 3 * density


def work(case):
    """State read and written once a step, every interacting pair's arithmetic once (about
    30 operations an LJ pair, 80 a Coulomb pair with erfc and exp)."""
    kind = case["kind"]
    if kind in ("step", "run", "config"):
        n = 4 * case["nx"] * case["ny"] * case["nz"] - case.get("missing", 0)
        pairs = n * _pairs_per_atom(case["density"], case["rc"])
        if kind == "config":
            return {"bytes": n * 2 * 24.0, "flops": 30 * pairs}
        steps = case["steps"]
        return {"bytes": n * (steps * 2 * 72.0 + 48), "flops": 30 * pairs * steps}
    if kind == "batch":
        t = np.random.default_rng(case["table"])
        n, pairs = 0, 0.0
        for _ in range(case["replicas"]):
            k = 4 * int(t.integers(case["small"], case["large"] + 1)) ** 3
            rho = float([0.1, 0.3, 0.5, 0.7, 0.8, 0.9][int(t.integers(0, 6))])
            t.uniform(1.0, 2.0)
            n, pairs = n + k, pairs + k * _pairs_per_atom(rho, 2.5)
        return {"bytes": n * (case["steps"] * 2 * 72.0 + 48), "flops": 30 * pairs * case["steps"]}
    if kind in ("water", "spce"):
        n = 3 * case["per_side"] ** 3
        flops = 80 * n * _pairs_per_atom(0.1, case["rc"])
        steps = case.get("steps", 1)
        if case.get("spacing", 0) > 0:  # 216 grid points a site, both ways, and two FFTs
            g = (case["per_side"] * 3.107 / case["spacing"]) ** 3
            flops += n * 216 * 8 + 2 * 2.5 * g * math.log2(g)
        else:  # eight real products a site serve four k vectors, twice over
            flops += n * 2.0 / 3.0 * math.pi * case["kmax"] ** 3 * 3 * 4
        return {"bytes": n * (steps * 2 * 72.0 if kind == "water" else 48.0), "flops": flops * steps}
    n = 4 * case["cells"] ** 3
    pairs = n * _pairs_per_atom(case["density"], 2.5)
    if kind == "adjoint":  # forward, recomputation and the second-order pass
        return {"bytes": n * case["steps"] * 3 * 2 * 72.0, "flops": 120 * pairs * case["steps"]}
    frame = 12 * n * _pairs_per_atom(case["density"], case["rmax"]) + 2 * n * 6.0
    return {"bytes": n * case["frames"] * (case["stride"] * 2 * 72.0 + 96),
            "flops": case["frames"] * (case["stride"] * 30 * pairs + frame)}


# ------------------------------------------------------------------- the same in 64 bits
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _fold(d, box):
    return d - box * torch.round(d / box)


def _near(pos, box, r):
    """Pairs (i, j), each once, with minimum-image distance below r."""
    n, dev = len(pos), pos.device
    dims = torch.floor(box / r).to(torch.int64)
    out_i, out_j = [], []
    if int(dims.min()) < 3 or n < 2000:
        for a in range(0, n, 1024):
            d = _fold(pos[a:a + 1024, None, :] - pos[None, :, :], box)
            i, j = torch.nonzero((d * d).sum(-1) < r * r, as_tuple=True)
            keep = i + a < j
            out_i.append(i[keep] + a)
            out_j.append(j[keep])
        return torch.cat(out_i), torch.cat(out_j)
    cell = torch.floor((pos / box + 0.5 - torch.floor(pos / box + 0.5)) * dims).to(torch.int64)
    cell = torch.minimum(cell, dims - 1)
    flat = (cell[:, 0] * dims[1] + cell[:, 1]) * dims[2] + cell[:, 2]
    count = torch.bincount(flat, minlength=int(dims.prod()))
    order = torch.argsort(flat, stable=True)
    start = torch.cumsum(count, 0) - count
    width = int(count.max())
    table = torch.full((int(dims.prod()), width), -1, dtype=torch.int64, device=dev)
    table[flat[order], torch.arange(n, device=dev) - start[flat[order]]] = order
    half = [(x, y, z) for x in (-1, 0, 1) for y in (-1, 0, 1) for z in (-1, 0, 1) if (x, y, z) >= (0, 0, 0)]
    for off in half:
        c = torch.remainder(cell + torch.tensor(off, device=dev), dims)
        other = (c[:, 0] * dims[1] + c[:, 1]) * dims[2] + c[:, 2]
        for a in range(0, n, 1 << 17):
            j = table[other[a:a + (1 << 17)]]
            i = torch.arange(a, a + len(j), device=dev)[:, None].expand_as(j)
            d = _fold(pos[i] - pos[j.clamp_min(0)], box)
            ok = (j >= 0) & ((d * d).sum(-1) < r * r)
            if off == (0, 0, 0):
                ok &= i < j
            out_i.append(i[ok])
            out_j.append(j[ok])
    return torch.cat(out_i), torch.cat(out_j)


def _scatter(n, i, j, f):
    out = torch.zeros((n, 3), dtype=F64, device=f.device)
    return out.index_add_(0, i, f).index_add_(0, j, -f)


def _lj(d, rc, shift, sigma=1.0, eps=1.0):
    """(u, w = r . F) of pairs at separation d; zero from rc on."""
    r2 = (d * d).sum(-1)
    s6 = (sigma * sigma / r2) ** 3
    u, w = 4.0 * eps * (s6 * s6 - s6), 24.0 * eps * (2.0 * s6 * s6 - s6)
    if shift:
        c6 = (sigma * sigma / (rc * rc)) ** 3
        uc, slope = 4.0 * eps * (c6 * c6 - c6), -24.0 * eps * (2.0 * c6 * c6 - c6) / rc
        r = torch.sqrt(r2)
        u, w = u - uc - (r - rc) * slope, w + r * slope
    inside = r2 < rc * rc
    zero = torch.zeros_like(u)
    return torch.where(inside, u, zero), torch.where(inside, w, zero), r2


class _LjForces:
    """LJ forces over a pair list that is renewed before a pair could be missed."""

    def __init__(self, box, rc, shift, skin=0.6):
        self.box, self.rc, self.shift, self.skin, self.at = box, rc, shift, skin, None

    def __call__(self, pos):
        if self.at is None or 2.0 * float(_fold(pos - self.at, self.box).norm(dim=1).max()) > self.skin:
            self.i, self.j = _near(pos, self.box, self.rc + self.skin)
            self.at = pos
        d = _fold(pos[self.i] - pos[self.j], self.box)
        u, w, r2 = _lj(d, self.rc, self.shift)
        return u.sum(), w.sum(), _scatter(len(pos), self.i, self.j, d * (w / r2)[:, None])


class _Chain:
    """A three-link Nose-Hoover chain, Suzuki-Yoshida weights of order four, three steps."""

    def __init__(self, dt, temp, tau, dof):
        self.dt, self.t, self.dof = dt, temp, dof
        self.q = [dof * temp * tau * tau, temp * tau * tau, temp * tau * tau]
        self.xi, self.p = [0.0] * 3, [0.0] * 3
        w = 1.0 / (2.0 - 2.0 ** (1.0 / 3.0))
        self.w = [w, 1.0 - 2.0 * w, w]

    def _link(self, j, ke, d):
        damp = math.exp(-0.25 * d * self.p[j + 1] / self.q[j + 1]) if j < 2 else 1.0
        g = (2.0 * ke - self.dof * self.t if j == 0
             else self.p[j - 1] ** 2 / self.q[j - 1] - self.t)
        self.p[j] = (self.p[j] * damp + 0.5 * d * g) * damp

    def half(self, ke):
        """Half a step: the factor for the velocities and the kinetic energy after it."""
        total = 1.0
        for w in self.w:
            d = w * 0.5 * self.dt
            for j in (2, 1, 0):
                self._link(j, ke, d)
            self.xi = [x + d * p / q for x, p, q in zip(self.xi, self.p, self.q)]
            f = math.exp(-d * self.p[0] / self.q[0])
            total, ke = total * f, ke * f * f
            for j in (0, 1, 2):
                self._link(j, ke, d)
        return total, ke

    def conserved(self):
        return (self.dof * self.t * self.xi[0] + self.t * (self.xi[1] + self.xi[2])
                + sum(0.5 * p * p / q for p, q in zip(self.p, self.q)))


def _trajectory(pos, vel, box, forces, steps, chain=None):
    """Velocity Verlet (inside a chain's halves): rows and the last state."""
    _, _, f = forces(pos)
    rows = []
    ke = 0.5 * float((vel * vel).sum())
    for _ in range(steps):
        if chain:
            scale, ke = chain.half(ke)
            vel = vel * scale
        vel = vel + 0.5 * DT * f
        pos = pos + DT * vel
        pos = pos - box * torch.floor(pos / box + 0.5)
        u, w, f = forces(pos)
        vel = vel + 0.5 * DT * f
        ke = 0.5 * float((vel * vel).sum())
        if chain:
            scale, ke = chain.half(ke)
            vel = vel * scale
        rows.append((float(u), float(w), ke, chain.conserved() if chain else 0.0))
    return np.array(rows), pos, vel, f


def _tensors(*arrays):
    return [torch.from_numpy(np.ascontiguousarray(a)).to(_device()) for a in arrays]


def _rows_out(rows, pos, vel):
    return {"energy": rows[..., 0], "virial": rows[..., 1], "kinetic": rows[..., 2],
            "conserved": rows[..., 3], "pos": pos.T.contiguous(), "vel": vel.T.contiguous()}


class _Spce:
    """Energy, virial trace and forces of SPC/E water: Ewald sums (k vectors or smooth PME
    of order 6), oxygen Lennard-Jones truncated with its analytic energy tail."""

    def __init__(self, case, box, m, dev):
        self.box, self.rc, self.n, self.m = box, case["rc"], 3 * m, m
        self.alpha = case["alpha"] if case["alpha"] > 0 else 5.6 / float(box.min())
        e = 1.602176565e-19
        self.c = e * e / (4.0 * math.pi * 8.854187817e-12) * 1e10 / 1.3806488e-23
        self.q = torch.from_numpy(_charges(m)).to(dev)
        self.volume = float(box.prod())
        self.at = None
        k = torch.arange(3 * m, device=dev).reshape(m, 3)
        self.bi, self.bj = k[:, [0, 0, 1]].reshape(-1), k[:, [1, 2, 2]].reshape(-1)
        self.grid = None
        if case.get("spacing", 0) > 0:
            self.grid = [md.fft_size(math.ceil(float(b) / case["spacing"])) for b in box]
            self._pme_setup(dev)
        else:
            r = torch.arange(-case["kmax"], case["kmax"] + 1, device=dev)
            v = torch.cartesian_prod(r, r, r)
            n2 = (v * v).sum(-1)
            half = (v[:, 0] > 0) | ((v[:, 0] == 0) & ((v[:, 1] > 0) | ((v[:, 1] == 0) & (v[:, 2] > 0))))
            self.k = 2.0 * math.pi * v[half & (n2 < case["kmax"] ** 2 + 2)].to(F64) / box

    def _pme_setup(self, dev):
        p = 6
        w = [0.0, 1.0]                      # M_2 at 0, 1
        for n in range(3, p + 1):           # M_p at the integers 0..p-1
            w = [(x * (w[x] if x < len(w) else 0.0) + (n - x) * (w[x - 1] if x else 0.0)) / (n - 1)
                 for x in range(n)]
        theta, freq = torch.ones((1, 1, 1), dtype=F64, device=dev), []
        for a, size in enumerate(self.grid):
            m = torch.arange(size, dtype=F64, device=dev)
            z = sum(w[k + 1] * torch.exp(2j * math.pi * m * k / size) for k in range(p - 1))
            shape = [1, 1, 1]
            shape[a] = size
            theta = theta / (z.abs() ** 2).reshape(shape)
            freq.append((torch.fft.fftfreq(size, 1.0 / size, dtype=F64, device=dev) / self.box[a]).reshape(shape))
        self.m2 = freq[0] ** 2 + freq[1] ** 2 + freq[2] ** 2
        safe = torch.where(self.m2 > 0, self.m2, torch.ones_like(self.m2))
        theta = theta * torch.exp(-(math.pi / self.alpha) ** 2 * safe) / safe
        self.theta = torch.where(self.m2 > 0, theta, torch.zeros_like(theta))

    def _weights(self, w):
        """M_6(w + j), j = 0..5, of fractions w."""
        zero = torch.zeros_like(w)
        c = [w, 1.0 - w]
        for n in range(3, 7):
            prev = c + [zero]
            c = [((w + j) * prev[j] + (n - j - w) * (prev[j - 1] if j else zero)) / (n - 1) for j in range(n)]
        return torch.stack(c, -1)

    def _pme(self, pos):
        pos = pos.detach().requires_grad_(True)
        size = torch.tensor(self.grid, device=pos.device)
        u = (pos / self.box - torch.floor(pos.detach() / self.box)) * size
        i0 = torch.floor(u.detach()).to(torch.int64)
        c = [self._weights(u[:, a] - i0[:, a]) for a in range(3)]
        j = torch.arange(6, device=pos.device)
        g = [torch.remainder(i0[:, a, None] - j, size[a]) for a in range(3)]
        flat = (g[0][:, :, None, None] * size[1] + g[1][:, None, :, None]) * size[2] + g[2][:, None, None, :]
        val = (self.q[:, None, None, None] * c[0][:, :, None, None] * c[1][:, None, :, None]
               * c[2][:, None, None, :])
        charge = torch.zeros(int(size.prod()), dtype=F64, device=pos.device)
        charge = charge.index_add(0, flat.reshape(-1), val.reshape(-1)).reshape(self.grid)
        f = torch.fft.fftn(charge)
        em = self.c / (2.0 * math.pi * self.volume) * self.theta * (f.real ** 2 + f.imag ** 2)
        energy = em.sum()
        (grad,) = torch.autograd.grad(energy, pos)
        virial = (em.detach() * (1.0 - 2.0 * (math.pi / self.alpha) ** 2 * self.m2)).sum()
        return energy.detach(), virial, -grad

    def _ksum(self, pos):
        k2 = (self.k * self.k).sum(-1)
        factor = 2.0 * self.c * (2.0 * math.pi / self.volume) * torch.exp(-k2 / (4.0 * self.alpha ** 2)) / k2
        e, w, f = 0.0, 0.0, torch.zeros_like(pos)
        for a in range(0, len(self.k), 1024):
            k, fac = self.k[a:a + 1024], factor[a:a + 1024]
            phase = pos @ k.T
            cs, sn = torch.cos(phase), torch.sin(phase)
            re, im = self.q @ cs, self.q @ sn
            em = fac * (re * re + im * im)
            e, w = e + em.sum(), w + (em * (1.0 - k2[a:a + 1024] / (2.0 * self.alpha ** 2))).sum()
            f = f + ((sn * (2.0 * fac * re) - cs * (2.0 * fac * im)) @ k) * self.q[:, None]
        return e, w, f

    def __call__(self, pos):
        if self.at is None or 2.0 * float((pos - self.at).norm(dim=1).max()) > 1.0:
            i, j = _near(pos, self.box, self.rc + 1.0)
            other = torch.div(i, 3, rounding_mode="floor") != torch.div(j, 3, rounding_mode="floor")
            self.i, self.j, self.at = i[other], j[other], pos
        a, n = self.alpha, self.n
        slope = 2.0 * a / math.sqrt(math.pi)
        i, j = self.i, self.j
        d = _fold(pos[i] - pos[j], self.box)
        r2 = (d * d).sum(-1)
        inside = r2 < self.rc ** 2
        i, j, d, r2 = i[inside], j[inside], d[inside], r2[inside]
        r = torch.sqrt(r2)
        cqq = self.c * self.q[i] * self.q[j]
        tail = torch.special.erfc(a * r) / r
        w = cqq * (slope * torch.exp(-a * a * r2) + tail)
        energy, virial = (cqq * tail).sum(), w.sum()
        oxy = (i % 3 == 0) & (j % 3 == 0)
        s6 = torch.where(oxy, (O_SIGMA ** 2 / r2) ** 3, torch.zeros_like(r2))
        lw = 24.0 * O_EPS * (2.0 * s6 * s6 - s6)
        energy, virial = energy + (4.0 * O_EPS * (s6 * s6 - s6)).sum(), virial + lw.sum()
        force = _scatter(n, i, j, d * ((w + lw) / r2)[:, None])
        sr3 = (O_SIGMA / self.rc) ** 3
        energy = energy + (8.0 / 3.0 * math.pi * self.m * (self.m / self.volume) * O_EPS * O_SIGMA ** 3
                           * (sr3 ** 3 / 3.0 - sr3))
        d = _fold(pos[self.bi] - pos[self.bj], self.box)
        r2 = (d * d).sum(-1)
        r = torch.sqrt(r2)
        cqq = self.c * self.q[self.bi] * self.q[self.bj]
        inner = torch.special.erf(a * r) / r
        w = cqq * (slope * torch.exp(-a * a * r2) - inner)
        energy, virial = energy - (cqq * inner).sum(), virial + w.sum()
        force = force + _scatter(n, self.bi, self.bj, d * (w / r2)[:, None])
        energy = energy - self.c * a / math.sqrt(math.pi) * (self.q * self.q).sum()
        e, w, f = self._pme(pos) if self.grid else self._ksum(pos)
        return energy + e, virial + w, force + f


def _bonds(x):
    """O-H1, O-H2, H1-H2 of (molecules, 3, 3) positions."""
    return torch.stack([x[:, 0] - x[:, 1], x[:, 0] - x[:, 2], x[:, 1] - x[:, 2]], 1)


def _spread(lam, bond, inv):
    """Displacements of the three sites for multipliers lam along the bonds."""
    g = lam[:, :, None] * bond
    return torch.stack([(g[:, 0] + g[:, 1]) * inv[0], (g[:, 2] - g[:, 0]) * inv[1],
                        (-g[:, 1] - g[:, 2]) * inv[2]], 1)


def _constrain(x, ref, inv, target2):
    """Positions on the constraint surface, corrections along the reference bonds
    (Newton on the three multipliers)."""
    ref = _bonds(ref)
    lam = torch.zeros((len(x), 3), dtype=F64, device=x.device)
    eye = torch.eye(3, dtype=F64, device=x.device)
    unit = [_bonds(_spread(eye[c].expand(len(x), 3), ref, inv)) for c in range(3)]
    for _ in range(8):
        b = _bonds(x + _spread(lam, ref, inv))
        jac = torch.stack([2.0 * (b * unit[c]).sum(-1) for c in range(3)], -1)
        lam = lam - torch.linalg.solve(jac, ((b * b).sum(-1) - target2)[..., None])[..., 0]
    return x + _spread(lam, ref, inv)


def _constrain_velocity(v, x, inv):
    b = _bonds(x)
    eye = torch.eye(3, dtype=F64, device=x.device)
    mat = torch.stack([(b * _bonds(_spread(eye[c].expand(len(x), 3), b, inv))).sum(-1) for c in range(3)], -1)
    lam = torch.linalg.solve(mat, -(b * _bonds(v)).sum(-1)[..., None])[..., 0]
    return v + _spread(lam, b, inv)


def _water_trajectory(case, pos, vel, box, mass):
    m = len(pos) // 3
    ff = _Spce(case, box, m, pos.device)
    dt, dof = _steps_tau(1.0), 6 * m - 3
    chain = _Chain(dt, 298.0, _steps_tau(100.0), dof) if case["thermostat"] else None
    inv = (1.0 / mass[:3]).tolist()
    hh = 2.0 * R_OH * math.sin(0.5 * ANGLE * math.pi / 180.0)
    target2 = torch.tensor([R_OH ** 2, R_OH ** 2, hh ** 2], dtype=F64, device=pos.device)
    kinetic = lambda v: 0.5 * float((mass[:, None] * v * v).sum())  # noqa: E731
    _, _, f = ff(pos)
    ke, rows = kinetic(vel), []
    for _ in range(case["steps"]):
        if chain:
            scale, ke = chain.half(ke)
            vel = vel * scale
        vel = vel + 0.5 * dt * f / mass[:, None]
        ref, free = pos.reshape(m, 3, 3), (pos + dt * vel).reshape(m, 3, 3)
        now = _constrain(free, ref, inv, target2)
        vel = vel + ((now - free) / dt).reshape(-1, 3)
        pos = now.reshape(-1, 3)
        u, w, f = ff(pos)
        vel = _constrain_velocity((vel + 0.5 * dt * f / mass[:, None]).reshape(m, 3, 3), now, inv).reshape(-1, 3)
        ke = kinetic(vel)
        if chain:
            scale, ke = chain.half(ke)
            vel = vel * scale
        rows.append((float(u), float(w), ke, chain.conserved() if chain else 0.0))
    if not case["thermostat"]:
        vel = vel * math.sqrt(298.0 / (2.0 * ke / dof))
    return _rows_out(np.array(rows), pos, vel)


def _adjoint_exact(case, pos, vel, box, grad):
    x, v = pos.clone().requires_grad_(True), vel.clone().requires_grad_(True)
    sigma = torch.ones((), dtype=F64, device=pos.device, requires_grad=True)
    eps = torch.ones((), dtype=F64, device=pos.device, requires_grad=True)
    i = j = at = None

    def forces(p):
        nonlocal i, j, at
        if at is None or 2.0 * float(_fold(p.detach() - at, box).norm(dim=1).max()) > 0.6:
            i, j = _near(p.detach(), box, 3.1)
            at = p.detach()
        d = _fold(p[i] - p[j], box)
        keep = (d.detach() ** 2).sum(-1) < 2.5 ** 2
        a, b = i[keep], j[keep]
        u, w, r2 = _lj(d[keep], 2.5, True, sigma, eps)
        f = d[keep] * (w / r2)[:, None]
        return u.sum(), w.sum(), torch.zeros_like(p).index_add(0, a, f).index_add(0, b, -f)

    rows, xx, vv = [], x, v
    _, _, f = forces(xx)
    for _ in range(case["steps"]):
        vv = vv + 0.5 * DT * f
        xx = xx + DT * vv
        u, w, f = forces(xx)
        vv = vv + 0.5 * DT * f
        rows.append(torch.stack([u, w, 0.5 * (vv * vv).sum()]))
    rows = torch.stack(rows)
    g = torch.autograd.grad((rows * grad).sum(), (eps, sigma, x, v))
    return {"rows": rows.detach(), "d_epsilon": np.float64(g[0].item()), "d_sigma": np.float64(g[1].item()),
            "d_pos": g[2], "d_vel": g[3]}


def _analysis_exact(case, pos, vel, box):
    forces = _LjForces(box, 2.5, False)
    bins, rmax = case["bins"], case["rmax"]
    hist = torch.zeros(bins, dtype=F64, device=pos.device)
    real, prev, frames, velocities = None, None, [], []
    for _ in range(case["frames"]):
        _, pos, vel, _ = _trajectory(pos, vel, box, forces, case["stride"])
        i, j = _near(pos, box, rmax)
        r = _fold(pos[i] - pos[j], box).norm(dim=1)
        hist += torch.bincount((r / (rmax / bins)).to(torch.int64), minlength=bins)[:bins].to(F64)
        real = pos if real is None else real + _fold(pos - prev, box)
        prev = pos
        frames.append(real)
        velocities.append(vel)
    msd, vacf = np.zeros(case["max_lag"] + 1), np.zeros(case["max_lag"] + 1)
    k = len(frames)
    for lag in range(min(k, case["max_lag"] + 1)):
        msd[lag] = np.mean([float(((frames[a + lag] - frames[a]) ** 2).sum(-1).mean()) for a in range(k - lag)])
        vacf[lag] = np.mean([float((velocities[a + lag] * velocities[a]).sum(-1).mean()) for a in range(k - lag)])
    edge = torch.arange(bins + 1, dtype=F64, device=pos.device) * (rmax / bins)
    n = len(pos)
    shell = 4.0 / 3.0 * math.pi * (edge[1:] ** 3 - edge[:-1] ** 3)
    g = 2.0 * hist / (k * n * (n / float(box.prod())) * shell)
    return {"histogram": None, "g": g, "msd": msd, "vacf": vacf / vacf[0],
            "pos": pos.T.contiguous(), "vel": vel.T.contiguous()}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("step", "run", "config"):
        if case.get("integrator") == "baoab":
            return None  # the noise is the generator's own
        pos, vel, box, temp = _lj_inputs(case, seed)
        n = len(pos)
        pos, vel, box = _tensors(pos, vel, box)
        forces = _LjForces(box, case["rc"], case["shift"])
        if kind == "config":
            e, w, f = forces(pos)
            return {"energy": np.float64(e.item()), "virial": np.float64(w.item()), "force": f.T.contiguous()}
        chain = _Chain(DT, temp, 0.5, 3 * n - 3) if case.get("integrator") == "nhc" else None
        rows, pos, vel, f = _trajectory(pos, vel, box, forces, case["steps"], chain)
        if kind == "step":
            return {"energy": rows[-1, 0], "virial": rows[-1, 1], "pos": pos.T.contiguous(),
                    "vel": vel.T.contiguous(), "force": f.T.contiguous()}
        return _rows_out(rows, pos, vel)
    if kind == "batch":
        all_rows, all_pos, all_vel = [], [], []
        for pos, vel, box, temp in _table(case, seed):
            n = len(pos)
            pos, vel, box = _tensors(pos, vel, box)
            rows, pos, vel, _ = _trajectory(pos, vel, box, _LjForces(box, 2.5, False), case["steps"],
                                            _Chain(DT, temp, 0.5, 3 * n - 3))
            all_rows.append(rows)
            all_pos.append(pos)
            all_vel.append(vel)
        return _rows_out(np.array(all_rows), torch.cat(all_pos), torch.cat(all_vel))
    if kind in ("water", "spce"):
        pos, vel, box, mass = _tensors(*_water(case["per_side"], _generator(seed)))
        if kind == "water":
            return _water_trajectory(case, pos, vel, box, mass)
        e, w, f = _Spce(case, box, len(pos) // 3, pos.device)(pos)
        return {"energy": np.float64(e.item()), "virial": np.float64(w.item()), "force": f.T.contiguous()}
    c = case["cells"]
    pos, vel, box = _lattice(c, c, c, case["density"], 0.722, _generator(seed))
    n = len(pos)
    pos, vel, box = _tensors(pos, vel, box)
    if kind == "adjoint":
        (grad,) = _tensors(_adjoint_weights(case, n, seed))
        return _adjoint_exact(case, pos, vel, box, grad)
    return _analysis_exact(case, pos, vel, box)
