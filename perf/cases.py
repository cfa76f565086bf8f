"""Performance cases of the particle engine: whole time steps in both particle
forms, the reference's staged time loop, the Poisson solve, a batched bias
sweep and the adjoint, each through the Python front end as a simulation
program calls it.

A state is an engine handle with a seeded particle load on a generated mesh;
a pass advances it (steps continue where the last pass stopped) and returns
what such a program reads after it: the charge density and the potential on
every dof, the kinetic energy, particle, absorbed and injected counts and the
objects' charge, current and potential of its steps.  The mixed form keeps its
particles and their weights in FP32, so its outputs are returned at that
precision; the FP64 form's are FP64.

A mesh (its host tables) is built once per geometry and shared by the states,
as in a program that sweeps seeds or biases over one mesh.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from puncpp_gb300 import _lib as L
from puncpp_gb300 import batch, meshgen, punc

ION_MASS = 1836.0
HALF, RADIUS = 10.0, 1.0     # the probe: [-10, 10]^3 around a unit sphere


def listed():
    return [
        # One time step of the smallest periodic box, its potential read back:
        # what a call costs when there is nearly nothing to compute (scripts
        # that advance step by step, tests, parameter scans of tiny boxes).
        dict(name="langmuir8-step-fp64", kind="step", mesh="langmuir", n=8, ppc=4, form="fp64", vth=0.0, field="dg0"),
        # The Langmuir oscillation of the benchmark (16^3 x 6 cells, 16
        # electrons per cell, cold, dt = 0.251), 20 steps between outputs.
        dict(name="langmuir16-fp64", kind="run", mesh="langmuir", n=16, ppc=16, form="fp64", vth=0.0, field="dg0",
             bz=0.0, steps=20),
        # A warm magnetised box of odd size in the mixed form.
        dict(name="langmuir21-mixed-b", kind="run", mesh="langmuir", n=21, ppc=7, form="mixed", vth=0.1, field="dg0",
             bz=1.0, steps=20),
        # The CG1 field (the reference time loop's default) in the FP64 form.
        dict(name="langmuir24-cg1-fp64", kind="run", mesh="langmuir", n=24, ppc=8, form="fp64", vth=0.1, field="cg1",
             bz=0.0, steps=10),
        # The reference's time loop call by call (distribute, solve_circuit,
        # field, boris, move, update, inject) around a small probe, FP64.
        dict(name="probe20-loop-fp64", kind="loop", mesh="probe", n=20, particles=200_000, form="fp64", field="cg1"),
        # The probe with the CG1 field in the mixed form, accel push.
        dict(name="probe33-cg1-mixed", kind="run", mesh="probe", n=33, particles=500_000, form="mixed", field="cg1",
             steps=10),
        # The probe at 40^3 with many particles per cell.
        dict(name="probe40-mixed", kind="run", mesh="probe", n=40, particles=3_000_000, form="mixed", field="dg0",
             steps=10),
        # The FP64 probe run at an odd, medium resolution.
        dict(name="probe53-fp64", kind="run", mesh="probe", n=53, particles=1_500_000, form="fp64", field="dg0",
             steps=10),
        # The probe run at 80^3 (3.1M cells, 2M + 2M particles), mixed form.
        dict(name="probe80-mixed", kind="run", mesh="probe", n=80, particles=4_000_000, form="mixed", field="dg0",
             steps=10),
        # A Poisson solve from a cold start, object at a fixed potential.
        dict(name="poisson56", kind="solve", mesh="probe", n=56),
        # A bias sweep of small independent runs in one engine.
        dict(name="batch24-mixed", kind="batch", runs=24, n_lo=8, n_hi=22, per_run=40_000, steps=10),
        # Gradients of a charge-density loss through 20 steps, checkpoints
        # every 5.
        dict(name="adjoint16", kind="adjoint", mesh="langmuir", n=16, particles=200_000, steps=20, every=5),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "run-periodic", "run-probe", "run-probe", "loop", "solve", "batch", "adjoint"])
    form = rng.choice(["fp64", "mixed"])
    field = rng.choice(["dg0", "dg0", "cg1"])
    if kind == "step":
        return dict(kind="step", mesh="langmuir", n=rng.randint(6, 24), ppc=rng.randint(1, 16), form=form,
                    vth=rng.choice([0.0, 0.1]), field=field)
    if kind == "run-periodic":
        return dict(kind="run", mesh="langmuir", n=rng.randint(8, 32), ppc=_log_int(rng, 1, 20), form=form,
                    vth=rng.choice([0.0, 0.05, 0.1]), field=field, bz=rng.choice([0.0, 1.0]),
                    steps=rng.randint(5, 20))
    if kind == "run-probe":
        return dict(kind="run", mesh="probe", n=_log_int(rng, 16, 72), particles=_log_int(rng, 40_000, 3_000_000),
                    form=form, field=field, steps=rng.randint(5, 10))
    if kind == "loop":
        return dict(kind="loop", mesh="probe", n=rng.randint(14, 32), particles=_log_int(rng, 20_000, 500_000),
                    form=form, field=field)
    if kind == "solve":
        return dict(kind="solve", mesh=rng.choice(["probe", "langmuir"]), n=rng.randint(12, 64))
    if kind == "batch":
        lo = rng.randint(7, 12)
        return dict(kind="batch", runs=rng.randint(2, 32), n_lo=lo, n_hi=lo + rng.randint(2, 14),
                    per_run=_log_int(rng, 5_000, 60_000), steps=rng.randint(5, 10))
    return dict(kind="adjoint", mesh="langmuir", n=rng.randint(8, 20), particles=_log_int(rng, 20_000, 250_000),
                steps=rng.randint(6, 20), every=rng.randint(2, 6))


# ---- meshes and loads ------------------------------------------------------

@functools.lru_cache(maxsize=16)
def _mesh(kind, n):
    ma = meshgen.langmuir_cube(n) if kind == "langmuir" else meshgen.probe_box(n, HALF, RADIUS)
    return punc.Mesh(ma)


@functools.lru_cache(maxsize=64)
def _probe_arrays(n, half, radius):
    return meshgen.probe_box(n, half, radius)


def _periodic_load(case, seed):
    """Electrons uniform in the unit cube (x displaced by 0.01 sin(2 pi x)),
    cold or thermal, weights of density 1 (omega_p = 1 with eps0 = 1)."""
    count = case["particles"] if "particles" in case else case["ppc"] * 6 * case["n"] ** 3
    rng = np.random.default_rng(seed)
    x = rng.random((count, 3))
    x[:, 0] = np.mod(x[:, 0] + 0.01 * np.sin(2 * np.pi * x[:, 0]), 1.0)
    # FP32 positions stay inside the box
    x = np.minimum(x, 1.0 - 1e-7)
    vth = case.get("vth", 0.1)
    v = rng.normal(0.0, vth, (count, 3)) if vth > 0 else np.zeros((count, 3))
    return x, v, 1.0 / count


def _probe_load(rng, half, radius, per_species):
    """(species, loads): electrons and ions of equal temperature at density 1
    (Debye length and plasma frequency 1), uniform over the box (points inside
    the object are dropped by the engine)."""
    volume = (2 * half) ** 3 - 4.0 / 3.0 * math.pi * radius ** 3
    w = volume / per_species
    species = [punc.Species(-w, w, n=1.0 / w, vth=1.0),
               punc.Species(w, ION_MASS * w, n=1.0 / w, vth=1.0 / math.sqrt(ION_MASS))]
    points = int(per_species * (2 * half) ** 3 / volume) + 1
    loads = [(half * (2.0 * rng.random((points, 3)) - 1.0), rng.normal(0.0, s.vth, (points, 3))) for s in species]
    return species, loads


def _form(case):
    return L.PG_MIXED if case["form"] == "mixed" else L.PG_FP64


def _held(case, a):
    """Outputs at the precision of the form's particles."""
    a = np.asarray(a, np.float64)
    return a.astype(np.float32) if case.get("form") == "mixed" else a


DT_PROBE, DT_PERIODIC = 0.05, 0.251


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return _prepare_batch(case, seed)
    mesh = _mesh(case["mesh"], case["n"])
    state = {"case": case, "mesh": mesh, "step": 0, "seed": seed, "objects": []}
    if kind == "solve":
        # every pass starts cold; the tolerances are the solver's defaults
        pop = punc.Population(mesh, periodic=case["mesh"] == "langmuir", warm_start=0, pcg_max_iter=4000)
        rho = punc.Function(pop, "rho")
        rho.set_local(_solve_rho(case, seed))
        state |= {"pop": pop, "rho": rho, "phi": punc.Function(pop, "phi"), "poisson": punc.PoissonSolver(pop),
                  "objects": [punc.Object(2, potential=-2.0)] if case["mesh"] == "probe" else []}
        return state
    if kind == "adjoint":
        x, v, w = _periodic_load(case, seed)
        pop = punc.Population(mesh, periodic=True, pcg_rtol=1e-12, pcg_atol=1e-30, pcg_max_iter=5000)
        pop.add_particles(x, v, -w, w)
        return state | {"pop": pop, "count": len(x), "target": _adjoint_target(case, seed)}
    mixed = case["form"] == "mixed"
    # the tolerances of the interaction program for the mixed form, the
    # solver's defaults for the FP64 form
    tol = dict(pcg_rtol=1e-10, pcg_atol=1e-12) if mixed else {}
    if case["mesh"] == "langmuir":
        x, v, w = _periodic_load(case, seed)
        pop = punc.Population(mesh, precision=_form(case), periodic=True, pcg_max_iter=4000, **tol)
        pop.add_particles(x, v, -w, w)
        return state | {"pop": pop, "dt": DT_PERIODIC, "inject": False, "phi": punc.Function(pop, "phi"),
                        "rho": punc.Function(pop, "rho")}
    rng = np.random.default_rng(seed)
    species, loads = _probe_load(rng, HALF, RADIUS, case["particles"] // 2)
    pop = punc.Population(mesh, precision=_form(case), capacity=int(1.5 * case["particles"]) + 65536,
                          pcg_max_iter=4000, **tol)
    for s, (x, v) in zip(species, loads):
        pop.add_particles(x, v, s.q, s.m)
    punc.create_flux(pop, species)
    objects = [punc.Object(2)]
    circuit = punc.CircuitCM(pop, objects, [(-1, 0, -2.0)], [], DT_PROBE)
    return state | {"pop": pop, "dt": DT_PROBE, "inject": True, "species": species, "objects": objects,
                    "circuit": circuit, "poisson": punc.PoissonSolver(pop), "esolver": punc.ESolver(pop),
                    "efield": punc.EFieldDG0(), "rho": punc.Function(pop, "rho"), "phi": punc.Function(pop, "phi"),
                    "E": punc.Function(pop, "E_cg1" if case["field"] == "cg1" else "E")}


def _prepare_batch(case, seed):
    rng = np.random.default_rng(seed)
    # geometry and biases belong to the sweep, not to the seed
    plan = np.random.default_rng(case["runs"] * 1000 + case["n_hi"])
    sides = plan.integers(case["n_lo"], case["n_hi"] + 1, case["runs"])
    halves = plan.uniform(2.5, 4.0, case["runs"])
    biases = plan.uniform(-5.0, 5.0, case["runs"])
    meshes = [_probe_arrays(int(n), float(h), 1.0) for n, h in zip(sides, halves)]
    b = batch.Batch(meshes, precision=L.PG_MIXED, capacity=int(2.0 * case["runs"] * case["per_run"]) + 65536,
                    pcg_rtol=1e-10, pcg_atol=1e-12, pcg_max_iter=4000)
    # one weight for the whole sweep, so the species are common to the runs
    w = float(np.mean((2 * halves) ** 3)) / (case["per_run"] // 2)
    species = [punc.Species(-w, w, n=1.0 / w, vth=1.0),
               punc.Species(w, ION_MASS * w, n=1.0 / w, vth=1.0 / math.sqrt(ION_MASS))]
    for r, h in enumerate(halves):
        count = int((2 * h) ** 3 / w)
        for s in species:
            b.add_particles(r, h * (2.0 * rng.random((count, 3)) - 1.0), rng.normal(0.0, s.vth, (count, 3)), s.q, s.m)
    b.create_flux(species, [seed * 1000 + r for r in range(case["runs"])])
    objects = b.objects()
    b.circuit(objects, biases, DT_PROBE)
    return {"case": dict(case, form="mixed", field="dg0"), "batch": b, "mesh": b.mesh, "pop": b.pop, "step": 0,
            "seed": 0, "objects": objects, "dt": DT_PROBE, "inject": True, "rho": punc.Function(b.pop, "rho"),
            "phi": punc.Function(b.pop, "phi")}


# ---- passes ----------------------------------------------------------------

def _object_values(case, objects):
    return _held(case, [[o.charge, o.current, o.potential] for o in objects])


def run(state):
    case, pop, kind = state["case"], state["pop"], state["case"]["kind"]
    if kind == "solve":
        return {"phi": state["poisson"].solve(state["phi"], state["rho"], state["objects"])}
    if kind == "adjoint":
        loss = punc.adjoint_forward(pop, [], 0.1, case["steps"], case["every"], state["target"], first_step=True,
                                    E0=(0.01, 0.0, 0.0), Ld=state["mesh"].Ld)
        grad_v, grad_e0, grad_x = punc.adjoint_backward(pop, state["count"])
        return {"loss": np.array([loss]), "grad_v": grad_v, "grad_e0": grad_e0, "grad_x": grad_x}
    if kind == "loop":
        return _loop(state)
    periodic = case.get("mesh") == "langmuir"
    args = dict(first_step=state["step"] == 0, Ld=state["mesh"].Ld if periodic else None, inject=state["inject"],
                seed=state["seed"], step_no=state["step"], efield_cg1=case["field"] == "cg1",
                B=(0.0, 0.0, case.get("bz", 0.0)), use_accel=not periodic and case["field"] == "cg1")
    if kind == "step":
        results = [punc.step(pop, state["objects"], state["dt"], **args)]
    else:
        results = punc.run_steps(pop, state["objects"], state["dt"], case["steps"], **args)
    state["step"] += len(results)
    out = {"phi": _held(case, state["phi"].vector()), "ke": _held(case, [r.KE for r in results]),
           "counts": np.array([[r.n_particles, r.n_absorbed, r.n_injected] for r in results], np.int64)}
    if kind != "step":
        out["rho"] = _held(case, state["rho"].vector())
    if state["objects"]:
        out["objects"] = _object_values(case, state["objects"])
    return out


def _loop(state):
    """One iteration of the reference's time loop."""
    case, pop, dt, objects = state["case"], state["pop"], state["dt"], state["objects"]
    rho = punc.distribute_cg1(pop, state["rho"])
    phi = state["poisson"].solve_circuit(state["phi"], state["rho"], state["mesh"], objects, state["circuit"])
    push_dt = dt * (0.5 if state["step"] == 0 else 1.0)
    if case["field"] == "cg1":
        field = state["esolver"].solve(state["E"], state["phi"])
        ke = punc.boris_cg1(pop, state["E"], (0.0, 0.0, 0.5), push_dt)
    else:
        state["efield"].solve(state["E"], state["phi"])
        field = state["E"].vector()
        ke = punc.boris(pop, state["E"], (0.0, 0.0, 0.5), push_dt)
    punc.move(pop, dt)
    pop.update(objects, dt)
    injected = punc.inject_particles(pop, state["species"], None, dt, seed=state["seed"], step=state["step"])
    state["step"] += 1
    return {"rho": _held(case, rho), "phi": _held(case, phi), "field": _held(case, field), "ke": _held(case, [ke]),
            "injected": np.array([injected, pop.num_of_particles()], np.int64),
            "objects": _object_values(case, objects)}


# ---- the least work of a pass ----------------------------------------------

def work(case):
    """Bytes: per step the particles' positions, velocities and cells read and
    written once and their species read, the cells' geometry, neighbours and
    dofs and the stiffness and mass matrices read once, the charge and the
    potential written once.  Operations: about 100 per particle and step, two
    per matrix entry."""
    kind = case["kind"]
    if kind == "batch":
        cells = case["runs"] * 6 * ((case["n_lo"] + case["n_hi"]) / 2) ** 3
        dofs, particles, real = cells / 6, case["runs"] * case["per_run"], 4
    else:
        cells, dofs = 6 * case["n"] ** 3, case["n"] ** 3
        particles = case.get("particles", case.get("ppc", 0) * cells)
        real = 4 if case.get("form") == "mixed" else 8
    steps = case.get("steps", 1) * (3 if kind == "adjoint" else 1)
    matrices = 12.0 * (7 + 15) * dofs
    per_step = particles * (12 * real + 9) + cells * (12 * real + 32) * min(1.0, particles / cells) + matrices + 32.0 * dofs
    return {"bytes": steps * per_step, "flops": steps * (100.0 * particles + 2 * 22 * dofs)}


# ---- the same in plain 64-bit torch ----------------------------------------

def exact(case, seed):
    """What the first pass of a new state returns, where the mesh allows a
    plain restatement: the periodic box (a uniform grid, where the P1 matrices
    are convolutions solved by FFT) and the Poisson solve on the probe mesh."""
    kind = case["kind"]
    if kind == "solve":
        return {"phi": _exact_periodic_solve(case, seed) if case["mesh"] == "langmuir" else _exact_probe_solve(case, seed)}
    if case.get("mesh") != "langmuir":
        return None
    if kind == "adjoint":
        return _exact_adjoint(case, seed)
    x, v, w = _periodic_load(case, seed)
    box = _PeriodicBox(case["n"])
    x, v = box.tensor(x), box.tensor(v)
    b = torch.tensor([0.0, 0.0, case.get("bz", 0.0)], dtype=torch.float64, device=box.device)
    steps, kes = case.get("steps", 1), []
    for k in range(steps):
        x, v, rho, phi, ke = box.step(x, v, w, DT_PERIODIC, k == 0, b, case["field"])
        kes.append(float(ke))
    out = {"phi": phi.cpu().numpy().ravel(), "ke": np.array(kes), "counts": None}
    if kind != "step":
        out["rho"] = rho.cpu().numpy().ravel()
    return out


class _PeriodicBox:
    """Particle-in-cell step on the unit cube of n^3 sub-cubes x 6 Kuhn
    tetrahedra, periodic, FP64."""

    PATHS = ((0, 1, 2), (0, 2, 1), (1, 0, 2), (1, 2, 0), (2, 0, 1), (2, 1, 0))

    def __init__(self, n):
        self.n, self.h = n, 1.0 / n
        self.device = "cuda" if torch.cuda.is_available() else "cpu"
        unit = torch.zeros((n, n, n), dtype=torch.float64, device=self.device)
        mass, stiff = unit.clone(), unit.clone()
        vol = self.h ** 3 / 6
        for path in self.PATHS:
            verts = [np.zeros(3, int)]
            for axis in path:
                verts.append(verts[-1] + np.eye(3, dtype=int)[axis])
            for a in verts:
                for c in verts:
                    d = tuple(int(t) % n for t in c - a)
                    mass[d] += vol / 20 * (2.0 if (a == c).all() else 1.0)
        for axis in range(3):
            for sign in (1, -1):
                d = [0, 0, 0]
                d[axis] = sign % n
                stiff[tuple(d)] -= self.h
        stiff[0, 0, 0] += 6 * self.h
        self.mass_hat = torch.fft.fftn(mass)
        stiff_hat = torch.fft.fftn(stiff).real
        stiff_hat[0, 0, 0] = 1.0
        self.green_hat = 1.0 / stiff_hat
        self.green_hat[0, 0, 0] = 0.0

    def tensor(self, a):
        return torch.as_tensor(a, dtype=torch.float64, device=self.device)

    def mass(self, u):
        # the stencils are symmetric: convolution and correlation agree
        return torch.fft.ifftn(torch.fft.fftn(u) * self.mass_hat).real

    def mass_inverse(self, u):
        return torch.fft.ifftn(torch.fft.fftn(u) / self.mass_hat).real

    def potential(self, rho):
        return torch.fft.ifftn(torch.fft.fftn(self.mass(rho)) * self.green_hat).real

    def locate(self, x):
        """Barycentric weights [P][4], flat dofs [P][4] and the axis order of
        each particle's tetrahedron."""
        s = x.detach() / self.h
        base = torch.floor(s).long()
        frac = x / self.h - base
        order = torch.argsort(frac.detach(), dim=1, descending=True)
        f = torch.gather(frac, 1, order)
        lam = torch.stack([1 - f[:, 0], f[:, 0] - f[:, 1], f[:, 1] - f[:, 2], f[:, 2]], dim=1)
        vert, dofs = base.clone(), []
        for k in range(4):
            if k:
                vert = vert.scatter_add(1, order[:, k - 1:k], torch.ones_like(order[:, :1]))
            w = torch.remainder(vert, self.n)
            dofs.append((w[:, 0] * self.n + w[:, 1]) * self.n + w[:, 2])
        return lam, torch.stack(dofs, dim=1), order

    def charge(self, x, w):
        lam, dofs, _ = self.locate(x)
        acc = torch.zeros(self.n ** 3, dtype=torch.float64, device=self.device)
        acc = acc.index_add(0, dofs.reshape(-1), (-w * lam).reshape(-1))
        return (acc / self.h ** 3).reshape((self.n,) * 3)

    def cell_field(self, x, phi):
        _, dofs, order = self.locate(x)
        p = phi.reshape(-1)[dofs]
        return torch.zeros_like(x).scatter(1, order, -(p[:, 1:] - p[:, :-1]) / self.h)

    def vertex_field(self, phi):
        rhs = torch.zeros((3,) + phi.shape, dtype=torch.float64, device=self.device)
        at = lambda u, d: torch.roll(u, shifts=[-int(t) for t in d], dims=(0, 1, 2))  # noqa: E731
        for path in self.PATHS:
            verts = [np.zeros(3, int)]
            for axis in path:
                verts.append(verts[-1] + np.eye(3, dtype=int)[axis])
            for k, axis in enumerate(path):
                part = -(at(phi, verts[k + 1]) - at(phi, verts[k])) / self.h * (self.h ** 3 / 24)
                for d in verts:
                    rhs[axis] += at(part, -d)
        return torch.stack([self.mass_inverse(r) for r in rhs])

    def step(self, x, v, w, dt, first, b, field, e0=None):
        rho = self.charge(x, w)
        phi = self.potential(rho)
        if field == "cg1":
            lam, dofs, _ = self.locate(x)
            ev = self.vertex_field(phi).reshape(3, -1)
            e = torch.stack([(lam * ev[c][dofs]).sum(1) for c in range(3)], dim=1)
        else:
            e = self.cell_field(x, phi)
        if e0 is not None:
            e = e + e0
        push = 0.5 * dt if first else dt
        half = -0.5 * push * e                      # q / m = -1
        mid = v + half
        ke = 0.5 * w * (mid * mid).sum()
        if b is not None and bool((b != 0).any()):
            t = torch.tan(-0.5 * push * b)
            s = 2 * t / (1 + (t * t).sum())
            rotated = mid + torch.cross(mid, t.expand_as(mid), dim=1)
            mid = mid + torch.cross(rotated, s.expand_as(mid), dim=1)
        v = mid + half
        x = x + dt * v
        x = x - torch.floor(x.detach())
        return x, v, rho, phi, ke


def _adjoint_target(case, seed):
    return 0.05 * np.random.default_rng(seed + 77).normal(0.0, 1.0, case["n"] ** 3)


def _exact_adjoint(case, seed):
    box = _PeriodicBox(case["n"])
    x, v, w = _periodic_load(case, seed)
    x0 = box.tensor(x).requires_grad_()
    v0 = box.tensor(v).requires_grad_()
    e0 = box.tensor([0.01, 0.0, 0.0]).requires_grad_()
    x, v = x0, v0
    for k in range(case["steps"]):
        x, v, _, _, _ = box.step(x, v, w, 0.1, k == 0, None, "dg0", e0)
    rho = box.charge(x, w).reshape(-1)
    loss = ((rho - box.tensor(_adjoint_target(case, seed))) ** 2).sum()
    loss.backward()
    return {"loss": np.array([float(loss.detach())]), "grad_v": v0.grad.cpu().numpy(), "grad_e0": e0.grad.cpu().numpy(),
            "grad_x": x0.grad.cpu().numpy()}


def _solve_rho(case, seed):
    """A charge density as the deposit gives it: particle noise on top of a
    smooth part."""
    mesh = _mesh(case["mesh"], case["n"]).arrays
    rng = np.random.default_rng(seed)
    if case["mesh"] == "langmuir":
        k = np.arange(case["n"]) / case["n"]
        smooth = np.broadcast_to(np.sin(2 * np.pi * k)[:, None, None], (case["n"],) * 3).ravel()
    else:
        smooth = np.exp(-np.abs(np.sqrt((mesh.coords ** 2).sum(1)) - RADIUS))
    return 0.1 * smooth + rng.normal(0.0, 0.3, mesh.n_dofs)


def _exact_periodic_solve(case, seed):
    box = _PeriodicBox(case["n"])
    return box.potential(box.tensor(_solve_rho(case, seed)).reshape((case["n"],) * 3)).cpu().numpy().ravel()


def _exact_probe_solve(case, seed):
    """P1 stiffness and mass matrices assembled from the mesh, Dirichlet values
    0 outside and -2 on the object, Jacobi-preconditioned CG to the attainable
    accuracy."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    ma = _mesh(case["mesh"], case["n"]).arrays
    coords = torch.as_tensor(ma.coords, dtype=torch.float64, device=dev)
    cells = torch.as_tensor(ma.cells, device=dev)
    n = ma.n_dofs
    p = coords[cells]
    jac = (p[:, 1:] - p[:, :1]).transpose(1, 2)               # columns: edges from vertex 0
    vol = torch.linalg.det(jac).abs() / 6
    grad = torch.linalg.inv(jac)                              # rows: grad lambda_1..3
    grad = torch.cat([-grad.sum(1, keepdim=True), grad], dim=1)
    stiff = torch.einsum("cid,cjd->cij", grad, grad) * vol[:, None, None]
    mass = (torch.ones(4, 4, dtype=torch.float64, device=dev) + torch.eye(4, dtype=torch.float64, device=dev)) / 20
    mass = mass[None] * vol[:, None, None]
    ij = torch.stack([cells[:, :, None].expand(-1, 4, 4).reshape(-1), cells[:, None, :].expand(-1, 4, 4).reshape(-1)])
    a = torch.sparse_coo_tensor(ij, stiff.reshape(-1), (n, n)).coalesce().to_sparse_csr()
    m = torch.sparse_coo_tensor(ij, mass.reshape(-1), (n, n)).coalesce().to_sparse_csr()
    fixed = torch.zeros(n, dtype=torch.bool, device=dev)
    value = torch.zeros(n, dtype=torch.float64, device=dev)
    tags = torch.as_tensor(ma.btags, device=dev)
    facets = torch.as_tensor(ma.bfacets, device=dev)
    for tag, u in ((2, -2.0), (1, 0.0)):
        at = facets[tags == tag].reshape(-1)
        fixed[at], value[at] = True, u
    free = (~fixed).double()
    b = (m @ torch.as_tensor(_solve_rho(case, seed), device=dev) - a @ value) * free
    diag = torch.zeros(n, dtype=torch.float64, device=dev)
    diag.index_add_(0, cells.reshape(-1), torch.diagonal(stiff, dim1=1, dim2=2).reshape(-1))
    u = torch.zeros_like(b)
    for _ in range(3):                                        # CG, then two refinements
        r = (b - a @ u) * free
        z = r / diag
        d, rz = z.clone(), r @ z
        stop = 1e-15 * float(b.norm())
        for _ in range(4000):
            if float(r.norm()) <= stop:
                break
            ad = (a @ d) * free
            alpha = rz / (d @ ad)
            u = u + alpha * d
            r = r - alpha * ad
            z = r / diag
            rz, old = r @ z, rz
            d = z + (rz / old) * d
    return (u + value).cpu().numpy()
