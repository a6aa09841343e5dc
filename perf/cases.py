"""What is timed: the time-step loop as a user's program drives it.

A case is one plasma deck and one way of driving it (``how``):

* ``run``    — ``Simulation.run`` for a stretch of steps (a write interval of the decks: 10), then what the loop's user
  reads there: potential, charge, density and field grids, kinetic and potential energies, particle counts (and the
  particle records of the smaller plasmas, or of a beam: its phase space);
* ``step``   — one ``Simulation.step`` call, then the same diagnostics: the smallest call;
* ``phases`` — one loop iteration method by method, as a main in the reference's style calls them;
* ``host``   — ``Simulation.run_host``: the particles live in the caller's pinned host buffers;
* ``batch``  — ``Batch.run``: many uneven runs advanced together;
* ``serve``  — ``Server``: requests submitted, served and collected.

Decks come from the repository's own workloads, or are generic plasmas of the same kind.
"""
from __future__ import annotations

import math
import os
import tempfile

import numpy as np
import torch

from epic2d_mcc_gb300 import api as E
from epic2d_mcc_gb300 import workloads as W

ME, AMU = W.ME, W.AMU
POISSON = {"dirichlet": "", "periodic": "poisson_bc = periodic\n", "dirichlet_x": "poisson_bc = dirichlet_x\n"}


# ------------------------------------------------------------------ cases ---
def _case(name, how, nx, ny, ppc, **kw):
    c = dict(name=name, how=how, nx=nx, ny=ny, ppc=ppc, plasma="two", solver="cg", tol=1e-10, omega=1.4,
             poisson="dirichlet", bc="pbc", shape="CIC", mixed=False, mcc=False, steps=1, particles=False, sort=-1,
             dt=0.01, te=1.0, grids=False, emitters=False, runs=0)
    unknown = set(kw) - set(c)
    if unknown:
        raise ValueError(unknown)
    c.update(kw)
    return c


def listed():
    return [
        # A single step call on the tests' deck size: latency, launches and host work.
        _case("step_cg_16", "step", 16, 16, 8, particles=True),
        # The plain FP64 periodic plasma (periodic_64) between two writes of its energies: SOR at omega 1.8.
        _case("run_sor_64", "run", 64, 64, 50, solver="gs", omega=1.8, tol=1e-8, poisson="periodic", steps=10,
              particles=True),
        # The headline FP64 deck with collisions (beam_mcc_256): PCG with phi = 0 on the x walls.
        _case("run_cg_beam_256", "run", 256, 256, 100, plasma="beam", poisson="dirichlet_x", mcc=True, steps=10),
        # A large FP64 plasma: the precision form's deck (twostream_1024) in the reference's arithmetic.
        _case("run_cg_1024", "run", 1024, 1024, 25, plasma="twostream", poisson="periodic", te=2.0, dt=0.05, steps=1),
        # The headline deck in mixed precision, one sort period.
        _case("run_mixed_beam_256", "run", 256, 256, 100, plasma="beam", poisson="dirichlet_x", mcc=True, mixed=True,
              steps=16),
        # The precision form (twostream_1024): 2.1e8 particles, the largest state.
        _case("run_mixed_1024", "run", 1024, 1024, 100, plasma="twostream", poisson="periodic", te=2.0, dt=0.05,
              mixed=True, steps=10, sort=32),
        # The reference's method sequence, method by method, on an odd rectangular grid with absorbing walls.
        _case("phases_cg_open_97x144", "phases", 97, 144, 30, bc="open", particles=True),
        # Conductors (conductors_64): SOR with the density override, absorbing walls, erasing push.
        _case("run_sor_conductors_64", "run", 64, 64, 100, solver="gs", omega=1.8, tol=1e-6, bc="open", te=2.0,
              grids=True, steps=5, particles=True),
        # Boltzmann electrons (gshybrid_64).
        _case("run_gshybrid_64", "run", 64, 64, 50, solver="gshybrid", omega=1.8, tol=1e-6, te=2.0, steps=5,
              particles=True),
        # Particles held by the caller in pinned host memory, every step's records there and back.
        _case("host_cg_128", "host", 128, 128, 50, steps=4),
        # Many uneven runs in one launch sequence, half of them colliding, one sort period.
        _case("batch_48", "batch", 256, 256, 0, runs=48, mixed=True, steps=16, sort=16),
        # A burst of served requests: grids of 64 to 256 cells a side, periodic and absorbing, half with collisions.
        _case("serve_24", "serve", 256, 256, 0, runs=24, mixed=True, steps=20),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    how = rng.choice(["run", "run", "run", "run", "step", "phases", "host", "batch", "serve"])
    if how in ("batch", "serve"):
        side = rng.choice([128, 192, 256])
        return {k: v for k, v in _case("", how, side, side, 0, runs=rng.randint(4, 40), mixed=True,
                                       steps=rng.randint(4, 24), sort=rng.choice([8, 16, 32])).items() if k != "name"}
    if how == "step":
        nx, ny = _log(rng, 8, 64), _log(rng, 8, 64)
    else:
        nx = _log(rng, 24, 400)
        ny = nx if rng.random() < 0.4 else max(16, min(400, int(nx * rng.uniform(0.5, 1.6))))
    mixed = how == "run" and rng.random() < 0.4
    solver = "cg"
    if not mixed and rng.random() < 0.35:
        solver = rng.choice(["gs", "gs", "gshybrid"])
    if solver != "cg":  # sweeps grow with the side: the sizes the SOR decks have
        nx, ny = min(nx, rng.randint(24, 100)), min(ny, rng.randint(24, 100))
    poisson = "dirichlet" if solver == "gshybrid" else rng.choice(["dirichlet", "periodic", "dirichlet_x"])
    bc = "pbc" if poisson != "dirichlet" else rng.choice(["pbc", "open", "reflective"])
    if solver == "gs" and poisson != "dirichlet":  # a wrapped lattice takes many more dependent steps a sweep
        nx, ny = min(nx, 72), min(ny, 72)
    mcc = how == "run" and solver != "gshybrid" and rng.random() < 0.3
    ppc = max(2, min(_log(rng, 4, 150), 6000000 // (nx * ny)))
    c = _case("", how, nx, ny, ppc, solver=solver, poisson=poisson, bc=bc, mixed=mixed, mcc=mcc,
              tol=rng.choice([1e-8, 1e-10]) if solver == "cg" else rng.choice([1e-6, 1e-8]),
              omega=1.4 if solver == "cg" else 1.8 if poisson != "dirichlet" else rng.choice([1.4, 1.8]),
              steps=1 if how in ("step", "phases") else rng.randint(2, 5) if solver != "cg" or how == "host" else
              rng.randint(2, 10),
              shape="NGP" if rng.random() < 0.15 else "CIC", te=rng.choice([0.5, 1.0, 2.0, 5.0]),
              plasma="beam" if mcc else rng.choice(["two", "two", "beam", "twostream"]) if solver != "gshybrid" else
              "two",  # collisions with 40 amu ions: the loop keeps ionisation products' ions at SI speeds
              particles=nx * ny * ppc <= 400000 and not mixed and not mcc,
              emitters=bc == "open" and solver == "cg" and how == "run" and rng.random() < 0.4)
    c["particles"] = c["particles"] and not c["emitters"]
    del c["name"]
    return c


# ------------------------------------------------------------------ decks ---
def _species(c, cells):
    """(name, mass, count, temp, charge, fract_den, drift) of each species."""
    n = cells * c["ppc"]
    ion, heavy = (float("%.8E" % m) for m in (1836 * ME, 40 * AMU))  # as the deck writes them
    if c["plasma"] == "beam":
        b = n // 10
        return [("electron", ME, n - b, c["te"], -1, 1.0, 0.0), ("ion", heavy, n, 0.026, 1, 0.0, 0.0),
                ("beam", ME, b, c["te"], -1, 1.0 / 9.0, 5.0)]
    if c["plasma"] == "twostream":
        vs = 3.0 * math.sqrt(2.0)
        return [("electron", ME, n // 2, c["te"], -1, 1.0, vs), ("ion", ion, n, 0.05, 1, 0.0, 0.0),
                ("beam", ME, n // 2, c["te"], -1, 1.0, -vs)]
    return [("electron", ME, n, c["te"], -1, 1.0, 0.0), ("ion", ion, n, 0.026, 1, 0.0, 0.0)]


def _deck(c):
    nx, ny = c["nx"], c["ny"]
    lines = ["%s,%.8E,%d,%g,%d,%.17g,%.17g,0,random" % (s[0], s[1], s[2], s[3], s[4], s[5], s[6])
             for s in _species(c, nx * ny)]
    extra = POISSON[c["poisson"]] + ("sor_omega = %g\n" % c["omega"] if c["solver"] != "cg" else "")
    text = W._TEMPLATE.format(num_ts=1000, dt=c["dt"], n=nx, solver=c["solver"], tol="%g" % c["tol"], maxit=200000,
                              solver_extra=extra, bc=c["bc"], coll="true" if c["mcc"] else "false", gas="1e20",
                              species="\n".join(lines))
    text = text.replace("Ny       = %d" % nx, "Ny       = %d" % ny, 1)
    text = text.replace("shapefunction = CIC", "shapefunction = %s" % c["shape"])
    if c["grids"]:
        text = W._sections(text, grids=[
            dict(type="reactconduct", min_x=nx * 18 // 64, max_x=nx * 21 // 64, min_y=ny * 12 // 64,
                 max_y=ny * 52 // 64, grid_voltage=10),
            dict(type="circular", x_center=nx * 42 // 64, y_center=ny // 2, electrode_number=6, grid_radius=10,
                 electrod_radius=2, electrode_voltage=-5)])
    if c["emitters"]:
        text = W._sections(text, emitters=[dict(x0=1, y0=ny // 8, x1=1, y1=ny - ny // 8, temp=0.5,
                                                numparticle=ny // 8 + 1, vdx=0.5, vdy=0, species_idx1=0, species_idx2=1)])
    return text


def _write(text):
    fd, path = tempfile.mkstemp(suffix=".ini", prefix="epic_case_")
    with os.fdopen(fd, "w") as f:
        f.write(text)
    return path


def _from_text(text, make):
    path = _write(text)
    try:
        return make(path)
    finally:
        os.unlink(path)


def _by_numpy(c):
    """Whether the particles are uploaded from host records (the plasmas of a few million particles at most)."""
    return not c["grids"] and c["nx"] * c["ny"] * c["ppc"] <= 900000


def _records(c, seed):
    """Uniform positions and Maxwellian velocities (units of the electrons' thermal speed) of every species."""
    rng = np.random.default_rng(seed)
    sp = _species(c, c["nx"] * c["ny"])
    scale = 1.0 / math.sqrt(sp[0][3] / sp[0][1])
    out = []
    for _, mass, n, temp, _, _, drift in sp:
        p = np.empty((n, 5))
        p[:, 0] = rng.random(n) * c["nx"]
        p[:, 1] = rng.random(n) * c["ny"]
        p[:, 2:] = rng.standard_normal((n, 3)) * (scale * math.sqrt(temp / mass))
        p[:, 2] += drift
        out.append(p)
    return out


# ---------------------------------------------------------------- prepare ---
class _State:
    pass


def prepare(case, seed):
    c = dict(case)
    s = _State()
    s.c = c
    _, ela, exc, ion = W.synthetic_table()
    s.table = (ela, exc, ion, 0.01, 1000.0)
    if c["how"] == "batch":
        sides = tuple(range(64, c["nx"] + 1, 16))
        reqs = [_from_text(d["ini"], lambda p, d=d: E.make_request(p, c["steps"], d["collisions"],
                                                                   1000003 * seed + d["seed"], precision=1))
                for d in W.batching_requests(seed=0, nruns=c["runs"], sides=sides)]
        s.batch = E.Batch(reqs, sort_every=c["sort"])
        s.batch.set_log_cross_sections(*s.table)
        s.batch.initial_field()
        return s
    if c["how"] == "serve":
        sides = tuple(x for x in (64, 128, 256) if x <= c["nx"])
        decks = W.serving_requests(seed=0, rate_per_s=1e4, window_s=1.0, sides=sides,
                                   step_scale=c["steps"] / 2750.0)[:c["runs"]]
        s.requests = [_from_text(d["ini"], lambda p, d=d: E.make_request(p, d["steps"], d["collisions"],
                                                                         1000003 * seed + d["seed"], 0.0,
                                                                         precision=1)) for d in decks]
        return s
    opts = {"seed": seed}
    if c["mixed"]:
        opts["precision"] = 1
    if c["sort"] >= 0:
        opts["sort_every"] = c["sort"]
    if c["mcc"] or c["emitters"]:  # room for the products and injections of many passes
        n = max(x[2] for x in _species(c, c["nx"] * c["ny"]))
        opts["capacity"] = n + n // 2 + (4000000 if c["emitters"] else 100000)
    s.sim = _from_text(_deck(c), lambda p: E.Simulation.from_ini(p, **opts))
    nsp = len(s.sim.species)
    if _by_numpy(c):
        recs = _records(c, seed)
        for k in range(nsp):
            s.sim.set_particles(k, recs[k])
    else:
        s.sim.load_particles_device(seed)
    if c["mcc"]:
        s.sim.set_log_cross_sections(*s.table)
    s.sim.initial_field()
    s.bufs, s.counts = {}, []
    for k in range(nsp):
        # every species, or the beam alone where a whole download would outweigh the loop it belongs to
        if c["particles"] or c["how"] == "host" or (c["plasma"] == "beam" and k == 2):
            n = s.sim.num_particles(k)
            n += n // 4 + 100000 if c["mcc"] or c["emitters"] else 0
            s.bufs[k] = torch.zeros((n, 5), dtype=torch.float64).pin_memory().numpy()
            s.counts.append(s.sim.particles_into(k, s.bufs[k]))
    s.sim.sync()
    return s


# -------------------------------------------------------------------- run ---
def _diagnostics(s):
    sim, c = s.sim, s.c
    nsp = len(sim.species)
    out = {"phi": sim.grid("phi"), "rho": sim.grid("rho"), "ke": [sim.compute_ke(k) for k in range(nsp)],
           "pe": sim.compute_pe(), "counts": [sim.num_particles(k) for k in range(nsp)]}
    if c["nx"] * c["ny"] <= 250000:
        out.update(den=[sim.den(k) for k in range(nsp)], efx=sim.grid("efx"), efy=sim.grid("efy"))
    if s.bufs:
        for k, b in s.bufs.items():
            sim.particles_into(k, b)
        out["particles"] = list(s.bufs.values())  # a species' records first; walls, conductors and MCC change their number
    return out


def run(s):
    c = s.c
    if c["how"] == "batch":
        s.batch.run(c["steps"])
        phi, rho = (np.concatenate([s.batch.grid(r, g) for r in range(c["runs"])]) for g in ("phi", "rho"))
        return {"phi": phi, "rho": rho, "n": s.batch.num_particles()}
    if c["how"] == "serve":
        srv = E.Server(60 << 30, max_inflight=8, chunk_steps=16)
        try:
            srv.set_log_cross_sections(*s.table)
            ids = [srv.submit(r) for r in s.requests]
            srv.start()
            srv.wait()
            res = [srv.result(i) for i in ids]
        finally:
            srv.close()
        return {"status": np.array([r.status for r in res]), "work": np.array([r.particle_steps for r in res]),
                "ke": np.array([r.kinetic_energy for r in res]), "pe": np.array([r.potential_energy for r in res])}
    sim = s.sim
    if c["how"] == "host":
        s.counts = sim.run_host(list(s.bufs.values()), s.counts, c["steps"], c["mcc"])
        return {"phi": sim.grid("phi"), "particles": list(s.bufs.values())}
    if c["how"] == "phases":
        nsp = len(sim.species)
        for k in range(nsp):
            sim.scatter_species(k)
        sim.compute_rho()
        iters, _, conv = sim.potential_solver()
        sim.calculate_efield()
        for k in range(nsp):
            sim.push_species(k)
        return dict(_diagnostics(s), iterations=iters, converged=conv)
    if c["how"] == "step":
        sim.step(c["mcc"])
    else:
        sim.run(c["steps"], c["mcc"])
    return _diagnostics(s)


# ------------------------------------------------------------------- work ---
def work(case):
    """Every step reads and writes each particle's stepped fields once (FP64: x, y, vx, vy; mixed: cell, two offsets,
    two velocities) and the node grids; about 60 operations a particle, and a fast direct field solve."""
    c = dict(case)
    if c["how"] == "batch":
        d = W.batching_requests(seed=0, nruns=c["runs"], sides=tuple(range(64, c["nx"] + 1, 16)))
        n, nodes, steps = sum(x["particles"] for x in d), sum(x["nx"] * x["ny"] for x in d), c["steps"]
    elif c["how"] == "serve":
        d = W.serving_requests(seed=0, rate_per_s=1e4, window_s=1.0, sides=tuple(x for x in (64, 128, 256) if x <= c["nx"]),
                               step_scale=c["steps"] / 2750.0)[:c["runs"]]
        n = sum(x["particles"] * x["steps"] for x in d) // c["steps"]
        nodes, steps = sum(x["side"] ** 2 * x["steps"] for x in d) // c["steps"], c["steps"]
    else:
        n = sum(s[2] for s in _species(c, c["nx"] * c["ny"]))
        nodes, steps = (c["nx"] + 1) * (c["ny"] + 1), c["steps"]
    per = 40 if c["mixed"] else 160 if c["how"] == "host" else 64
    return {"bytes": float(steps * (per * n + 40 * nodes)),
            "flops": float(steps * (60 * n + 20 * nodes * math.log2(max(nodes, 2))))}


# ------------------------------------------------------------------ exact ---
def _basis(n, periodic):
    """Orthonormal symmetric eigenvectors of the second difference on n points, and its eigenvalues."""
    if periodic:
        j = np.arange(n)
        a = 2 * np.pi * (np.outer(j, j) % n) / n
        return (np.cos(a) + np.sin(a)) / math.sqrt(n), -4 * np.sin(np.pi * j / n) ** 2
    j = np.arange(1, n + 1)
    return (math.sqrt(2 / (n + 1)) * np.sin(np.pi * (np.outer(j, j) % (2 * (n + 1))) / (n + 1)),
            -4 * np.sin(np.pi * j / (2 * (n + 1))) ** 2)


class _Loop:
    """The loop in plain numpy, FP64, unit cells, with direct field solves (periodic or absorbing walls, CIC)."""

    def __init__(self, c, seed):
        self.c = c
        qe, eps0 = 1.602176565e-19, 8.85418782e-12
        sp = _species(c, c["nx"] * c["ny"])
        dens = 1e13
        norm = [0.0] * len(sp)
        norm[1] = dens
        norm[0] = dens / sum(-s[4] * s[5] for s in sp)
        for i in range(2, len(sp)):
            norm[i] = sp[i][5] * norm[0]
        kt = [s[3] * qe for s in sp]
        lde = math.sqrt(eps0 * kt[0] / (norm[0] * qe * qe))
        wpe = math.sqrt(norm[0] * qe * qe / (ME * eps0))
        self.dt = c["dt"]
        self.src = 1.0  # (L / LDe)^2
        vn = lde * wpe
        self.qmk = [s[4] * qe / s[1] * (dens * qe * lde) / (eps0 * wpe * vn) for s in sp]
        nx, ny = c["nx"] + 1, c["ny"] + 1
        self.w = [norm[i] * c["nx"] * c["ny"] / s[2] / dens for i, s in enumerate(sp)]
        self.q = [s[4] for s in sp]
        self.nx, self.ny = nx, ny
        self.parts = _records(c, seed)
        self.unit = [0.5 * s[1] * vn * vn for s in sp]
        self.spwt = [norm[i] * c["nx"] * c["ny"] * lde * lde / s[2] for i, s in enumerate(sp)]
        self.th = sp[0][3] * qe * self.spwt[0] * sp[0][2]
        self.pe_unit = 0.5 * eps0 * lde * lde * (dens * qe * lde / eps0) ** 2 / self.th
        mode = c["poisson"]
        if mode == "dirichlet" and c["solver"] == "cg":  # the flattened node vector, rows of nx
            self.R, self.C, wr, wc = ny, nx, False, False
        elif mode == "dirichlet":
            self.R, self.C, wr, wc = nx - 2, ny - 2, False, False
        else:
            wr = mode == "periodic"
            self.R, self.C, wc = nx - 1 - (not wr), ny - 1, True
        qr, lr = _basis(self.R, wr)
        qc, lc = _basis(self.C, wc)
        lam = lr[:, None] + lc[None, :]
        if mode == "periodic":
            lam[0, 0] = 1.0
        self.bases = qr, qc, lam
        px = c["bc"] == "pbc" if mode == "dirichlet" else mode == "periodic"
        py = c["bc"] == "pbc" if mode == "dirichlet" else True
        self.edges = px, py
        self.field()
        for p, qmk in zip(self.parts, self.qmk):
            e = self.gather(p)
            p[:, 2] -= 0.5 * qmk * e[0] * self.dt
            p[:, 3] -= 0.5 * qmk * e[1] * self.dt

    def nodes(self, p):
        i, j = p[:, 0].astype(np.int64), p[:, 1].astype(np.int64)
        a, b = p[:, 0] - i, p[:, 1] - j
        k = i * self.ny + j
        return ((k, (1 - a) * (1 - b)), (k + self.ny, a * (1 - b)), (k + 1, (1 - a) * b), (k + self.ny + 1, a * b))

    def gather(self, p):
        at = self.nodes(p)
        return [sum(f.ravel()[k] * w for k, w in at) for f in (self.ex, self.ey)]

    def field(self):
        nx, ny, c = self.nx, self.ny, self.c
        rho = np.zeros((nx, ny))
        self.den = []
        for p, w, q in zip(self.parts, self.w, self.q):
            d = sum(np.bincount(k, weights=wt, minlength=nx * ny) for k, wt in self.nodes(p)).reshape(nx, ny) * w
            if c["bc"] == "pbc":
                d[:, 0] += d[:, -1]
                d[:, -1] = d[:, 0]
                d[0] += d[-1]
                d[-1] = d[0]
            else:
                d[:, 0] *= 0.5
                d[:, -1] *= 0.5
                d[0] *= 0.5
                d[-1] *= 0.5
            rho += q * d
            self.den.append(d)
        self.rho = rho
        mode, R, C = c["poisson"], self.R, self.C
        b = -rho
        phi = np.zeros((nx, ny))
        qr, qc, lam = self.bases
        if mode == "dirichlet" and c["solver"] == "cg":
            b = b.copy()
            b[0] = b[-1] = 0
            b[:, 0] = b[:, -1] = 0
            b = b.reshape(R, C)
        elif mode == "dirichlet":
            b = b[1:-1, 1:-1]
        else:
            b = b[nx - 1 - R:nx - 1, :C]
            if mode == "periodic":
                b = b - b.mean()
        t = (qr @ b @ qc) / lam
        if mode == "periodic":
            t[0, 0] = 0.0
        x = qr @ t @ qc
        if mode == "dirichlet" and c["solver"] == "cg":
            phi = x.reshape(nx, ny)
        elif mode == "dirichlet":
            phi[1:-1, 1:-1] = x
        else:
            phi[nx - 1 - R:nx - 1, :C] = x
            phi[:, -1] = phi[:, 0]
            if mode == "periodic":
                phi[-1] = phi[0]
        self.phi = phi
        self.ex, self.ey = self.slope(phi, self.edges[0]), self.slope(phi.T, self.edges[1]).T

    @staticmethod
    def slope(f, periodic):
        e = np.empty_like(f)
        e[1:-1] = -(f[2:] - f[:-2]) / 2
        if periodic:
            e[0] = e[-1] = -(f[1] - f[-2]) / 2
        else:
            e[0], e[-1] = -(f[1] - f[0]), -(f[-1] - f[-2])
        return e

    def step(self):
        lx, ly = float(self.nx - 1), float(self.ny - 1)
        self.field()
        for s, p in enumerate(self.parts):
            e = self.gather(p)
            p[:, 2] += self.qmk[s] * e[0] * self.dt
            p[:, 3] += self.qmk[s] * e[1] * self.dt
            p[:, 0] += p[:, 2] * self.dt
            p[:, 1] += p[:, 3] * self.dt
            if self.c["bc"] == "pbc":
                for a, l in ((0, lx), (1, ly)):
                    p[:, a] = np.where(p[:, a] < 0, p[:, a] + l, np.where(p[:, a] >= l, p[:, a] - l, p[:, a]))
            else:
                self.parts[s] = p[(p[:, 0] >= 0) & (p[:, 0] < lx) & (p[:, 1] >= 0) & (p[:, 1] < ly)]


def exact(case, seed):
    c = dict(case)
    if (c["how"] in ("batch", "serve") or not _by_numpy(c) or c["mcc"] or c["grids"] or c["emitters"]
            or c["solver"] == "gshybrid" or c["shape"] != "CIC" or c["bc"] == "reflective"
            or c["nx"] * c["ny"] * c["ppc"] * (c["steps"] + 1) > 8000000):
        return None
    loop = _Loop(c, seed)
    for _ in range(c["steps"]):
        loop.step()
    if c["how"] == "host":
        return {"phi": loop.phi.ravel(), "particles": loop.parts}
    out = {"phi": loop.phi.ravel(), "rho": loop.rho.ravel(),
           "ke": [loop.spwt[k] * loop.unit[k] * (p[:, 2:] ** 2).sum(axis=0) / loop.th for k, p in enumerate(loop.parts)],
           "pe": float(loop.pe_unit * ((loop.ex ** 2 + loop.ey ** 2).sum())), "counts": [None] * len(loop.parts),
           "den": [d.ravel() for d in loop.den], "efx": loop.ex.ravel(), "efy": loop.ey.ravel()}
    if c["bc"] == "pbc" and (c["particles"] or c["plasma"] == "beam"):
        out["particles"] = loop.parts if c["particles"] else loop.parts[2:]
    if c["how"] == "phases":
        out["iterations"] = None
        out["converged"] = None
    return out
