"""Timed cases of the lattice-Boltzmann step: what a program that uses this library has it do.

Four kinds of work, each through the public Python binding:

  fluid    a lattice is advanced `steps` time steps, then its macroscopic fields
           are read into device arrays (what a program does between two reports)
  report   the same, with the report itself: residual and means
           (`treat_data`) and the fields in host memory (`macroscopics`)
  spheres  the same with movable spheres in the fluid (immersed boundary)
  serving  a server takes a mix of duct requests of uneven sizes, some with
           spheres, runs them to their step counts and hands back each field

`exact` restates the same physics in 64-bit torch (collision, streaming,
half-way bounce-back, moving lid, Power-Law and Bingham relaxation, Peskin
interpolation, direct forcing and spreading), without the library.
"""
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "viscoplastic-lbm_b200"))
import vlbm  # noqa: E402

# Velocity sets: the library's population order (rest, then opposite pairs).
C27 = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 0), (-1, -1, 0),
       (1, 0, 1), (-1, 0, -1), (0, 1, 1), (0, -1, -1), (1, -1, 0), (-1, 1, 0), (1, 0, -1), (-1, 0, 1), (0, 1, -1),
       (0, -1, 1), (1, 1, 1), (-1, -1, -1), (1, 1, -1), (-1, -1, 1), (1, -1, 1), (-1, 1, -1), (-1, 1, 1), (1, -1, -1)]
WEIGHTS = {19: (1 / 3, 1 / 18, 1 / 36), 27: (8 / 27, 2 / 27, 1 / 54, 1 / 216)}

BUILDERS = {"plates": vlbm.BUILDER_PLATES_Y, "duct": vlbm.BUILDER_DUCT_YZ, "box": vlbm.BUILDER_CLOSED_BOX,
            "cavity": vlbm.BUILDER_LID_CAVITY_CLOSED}
WALLS = {"plates": (0, 1, 0), "duct": (0, 1, 1), "box": (1, 1, 1), "cavity": (1, 1, 1)}   # axes with walls
STORAGE = {"f32": vlbm.STORE_F32, "f16": vlbm.STORE_F16}
RHEOLOGY = {"newtonian": vlbm.NEWTONIAN, "bingham": vlbm.BINGHAM, "powerlaw": vlbm.POWERLAW}
OPERATOR = {"regularized": vlbm.OP_REGULARIZED, "bgk": vlbm.OP_BGK}


def case(kind, name, **kw):
    c = dict(kind=kind, vel_set=19, operator="regularized", rheology="bingham", storage="f32", walls="plates",
             n_index=1.0, nx=64, ny=64, nz=64, steps=50)
    c.update(kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # a small verification run: Newtonian BGK Poiseuille channel; launches and latency count
        case("fluid", "poiseuille_64x32x32", operator="bgk", rheology="newtonian", nx=64, ny=32, nz=32, steps=100),
        # the headline lattice of the benchmark, in both storage types
        case("fluid", "channel_256x128x64_f32", nx=256, ny=128, nz=64, steps=50),
        case("fluid", "channel_256x128x64_f16", storage="f16", nx=256, ny=128, nz=64, steps=50),
        # a production lattice in half storage
        case("fluid", "channel_256_f16", storage="f16", nx=256, ny=256, nz=256, steps=20),
        # the largest configuration: D3Q27 shear-thinning lid-driven cavity, single precision
        case("fluid", "cavity_256_q27_f32", vel_set=27, rheology="powerlaw", n_index=0.5, walls="cavity",
             nx=256, ny=256, nz=256, steps=20),
        # an odd, ragged lattice: shear-thickening cavity in half storage
        case("fluid", "cavity_ragged_q27_f16", vel_set=27, rheology="powerlaw", n_index=1.5, walls="cavity",
             storage="f16", nx=101, ny=90, nz=75, steps=50),
        # one duct of the serving stream, alone
        case("fluid", "duct_144x56x56_q27_f16", vel_set=27, walls="duct", storage="f16", nx=144, ny=56, nz=56,
             steps=100),
        # a report: steps, residual and means, the fields in host memory
        case("report", "report_128x96x64_f32", nx=128, ny=96, nz=64, steps=50),
        # the settling suspension: 64 spheres, three forcing iterations
        case("spheres", "suspension_192x192x384", walls="box", nx=192, ny=192, nz=384, steps=10, spheres=64,
             radius=8.0, iterations=3),
        # a serving-size duct with a few spheres
        case("spheres", "duct_4_spheres_f16", walls="duct", storage="f16", nx=144, ny=56, nz=56, steps=50, spheres=4,
             radius=5.0, iterations=1),
        # the serving loop: a mix of requests through 16 slots
        {"kind": "serving", "name": "serving_32_requests", "requests": 32, "slots": 16, "mix": 7, "most": 96,
         "steps": 300},
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["fluid"] * 6 + ["report"] + ["spheres"] * 2 + ["serving"])
    if kind == "serving":
        return {"kind": "serving", "requests": rng.randint(8, 32), "slots": rng.choice([8, 16, 32]),
                "mix": rng.randrange(1 << 20), "most": rng.randint(40, 96), "steps": rng.randint(100, 300)}
    storage = rng.choice(["f32", "f16"])
    if kind == "spheres":
        n, r = log_int(1, 64), rng.choice([4.0, 5.0, 6.0, 8.0])
        side = int(math.ceil((2 * r + 4) * (n ** (1 / 3) + 1) * 1.1))   # room for a loose packing
        nx, ny, nz = (min(256, max(32, int(side * rng.uniform(1.0, 1.5)))) for _ in range(3))
        return case(kind, None, walls=rng.choice(["duct", "box"]), vel_set=rng.choice([19, 27]), storage=storage,
                    nx=nx, ny=ny, nz=nz, spheres=n, radius=r, iterations=rng.randint(1, 3), steps=10)
    rheology = rng.choice(["newtonian", "bingham", "powerlaw"])
    nx, ny, nz = log_int(24, 256), log_int(16, 256), log_int(16, 256)
    if rng.random() < 0.4:
        nx = max(32, nx // 32 * 32)
    most = 100 if kind == "fluid" else 50
    return case(kind, None, vel_set=rng.choice([19, 27]), operator=rng.choice(["regularized", "regularized", "bgk"]),
                rheology=rheology, n_index=rng.choice([0.5, 1.0, 1.5, 0.8]) if rheology == "powerlaw" else 1.0,
                storage=storage, walls=rng.choice(["plates", "duct", "cavity"]), nx=nx, ny=ny, nz=nz,
                steps=max(10, min(most, int(3.0e8 / (nx * ny * nz)))))


# ------------------------------------------------------------------ physics --
def physics(c):
    """Rheology and driving of a case, in lattice units."""
    p = dict(tau=0.9, eta_p=0.1, yield_stress=1e-5, n_index=c["n_index"], k=0.0, lid=0.0, f=(0.0, 0.0, 0.0))
    if c["walls"] in ("plates", "duct"):
        p["f"] = (5e-6, 0.0, 0.0) if c["rheology"] != "newtonian" else (1e-6, 0.0, 0.0)
    if c["walls"] == "cavity":
        p["lid"] = 0.05
    if c["rheology"] == "powerlaw":
        n, side = c["n_index"], min(c["nx"], c["ny"])
        p["k"] = 0.05 ** (2.0 - n) * side ** n / min(400.0, 2.0 * side)   # Re = U^(2-n) L^n / K
    return p


def config(c):
    p = physics(c)
    kw = dict(nx=c["nx"], ny=c["ny"], nz=c["nz"], vel_set=c["vel_set"], collision=OPERATOR[c["operator"]],
              rheology=RHEOLOGY[c["rheology"]], storage=STORAGE[c["storage"]], fx=p["f"][0], fy=p["f"][1],
              fz=p["f"][2])
    if c["rheology"] == "newtonian":
        kw.update(tau=p["tau"])
    elif c["rheology"] == "bingham":
        kw.update(eta_p=p["eta_p"], yield_stress=p["yield_stress"])
    else:
        kw.update(n_index=p["n_index"], k_consistency=p["k"], gamma0=0.0)
    if p["lid"]:
        kw.update(ux_bc=[0, p["lid"]])
    return vlbm.Config.default(**kw)


def device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def velocity_field(c, seed):
    """Density and velocity [nz][ny][nx], a few long waves that vanish at the walls."""
    rng = random.Random(seed * 7919 + 13)
    n = (c["nz"], c["ny"], c["nx"])
    wall = WALLS[c["walls"]][::-1]
    axes = [(torch.arange(m, device=device(), dtype=torch.float64) + 0.5) / m for m in n]
    shape = ((-1, 1, 1), (1, -1, 1), (1, 1, -1))
    out = []
    for amplitude in (0.002, 0.02, 0.02, 0.02):   # rho - 1, ux, uy, uz
        field = torch.zeros(n, device=device(), dtype=torch.float64)
        for _ in range(3):
            term = torch.full((1, 1, 1), amplitude / 3, device=device(), dtype=torch.float64)
            for a in range(3):
                k, phase = rng.randint(1, 3), rng.uniform(0, 2 * math.pi)
                wave = torch.sin(math.pi * k * axes[a]) if wall[a] else torch.sin(2 * math.pi * k * axes[a] + phase)
                term = term * wave.view(shape[a])
            field += rng.uniform(0.5, 1.0) * rng.choice([-1, 1]) * term
        out.append(field)
    return out[0] + 1.0, out[1], out[2], out[3]


def populations(c, seed):
    """Initial populations [Q][nz][ny][nx] in single precision: equilibrium of the field above."""
    rho, ux, uy, uz = velocity_field(c, seed)
    uu = ux * ux + uy * uy + uz * uz
    f = torch.empty((c["vel_set"],) + tuple(rho.shape), device=device(), dtype=torch.float32)
    for i, (cx, cy, cz) in enumerate(C27[:c["vel_set"]]):
        cu = cx * ux + cy * uy + cz * uz
        f[i] = weight(c["vel_set"], i) * rho * (1 + 3 * cu + 4.5 * cu * cu - 1.5 * uu)
    return f


def weight(q, i):
    return WEIGHTS[q][sum(abs(v) for v in C27[i])]


def sphere_set(c, seed):
    """Sphere records of a case: centres two units apart and two from the walls, moving and spinning slowly."""
    rng = random.Random(seed * 104729 + 5)
    r, n, wall = c["radius"], (c["nx"], c["ny"], c["nz"]), WALLS[c["walls"]]
    out = []
    for _ in range(c["spheres"]):
        for _try in range(20000):
            p = [rng.uniform(r + 2, m - 1 - r - 2) if w else rng.uniform(0, m) for m, w in zip(n, wall)]
            far = True
            for o in out:
                d = [abs(a - b) for a, b in zip(p, o[:3])]
                d = [v if w else min(v, m - v) for v, m, w in zip(d, n, wall)]
                far = far and sum(v * v for v in d) >= (2 * r + 2) ** 2
            if far:
                break
        else:
            break   # no room for another one
        out.append(p + [rng.uniform(-2e-3, 2e-3) for _ in range(3)] + [rng.uniform(-2e-4, 2e-4) for _ in range(3)])
    return out


def ibm_config(c):
    w = WALLS[c["walls"]]
    return vlbm.IbmConfig.default(max_iterations=c["iterations"], gx=0.0, gy=0.0, gz=-1e-5, wall_x=w[0], wall_y=w[1],
                                  wall_z=w[2], particle_young=1e5, wall_young=1e5, particle_poisson=0.3,
                                  wall_poisson=0.3, pp_friction=0.3, pw_friction=0.3)


def uniform_flow(seed):
    rng = random.Random(seed * 31 + 3)
    return [rng.uniform(-5e-3, 5e-3) for _ in range(3)]


def requests(c, seed):
    """The serving mix: sizes and step counts belong to the case, the fluids and spheres to the seed."""
    size, rng = random.Random(c["mix"]), random.Random(seed * 65537 + 1)
    out = []
    for tag in range(c["requests"]):
        nx, ny = size.randint(32, 256), size.randint(16, c["most"])
        q, tau, bn = size.choice([19, 27]), rng.uniform(0.6, 1.2), 10 ** rng.uniform(-1, 1)
        steps, carries = int(c["steps"] * size.uniform(0.5, 1.5)), size.random() < 0.2
        nu, u, h = (tau - 0.5) / 3.0, 0.02, ny - 2
        cfg = vlbm.Config.default(nx=nx, ny=ny, nz=ny, vel_set=q, collision=vlbm.OP_REGULARIZED,
                                  rheology=vlbm.BINGHAM, eta_p=nu, yield_stress=bn * nu * u / h,
                                  fx=8.0 * nu * u / (h * h), storage=vlbm.STORE_F16)
        spheres = []
        if carries and ny >= 24:
            c1 = dict(nx=nx, ny=ny, nz=ny, walls="duct", radius=5.0, spheres=size.randint(1, 4))
            spheres = sphere_set(c1, seed * 131 + tag)
        out.append(dict(tag=tag, cfg=cfg, steps=steps, spheres=spheres, radius=5.0))
    return out


def sphere_records(rows, radius):
    return [vlbm.Sphere(diameter=2 * radius, cx=r[0], cy=r[1], cz=r[2], vx=r[3], vy=r[4], vz=r[5], wx=r[6], wy=r[7],
                        wz=r[8], density=1.5, movable=1) for r in rows]


# ------------------------------------------------------------------ running --
def prepare(c, seed):
    if c["kind"] == "serving":
        reqs = requests(c, seed)
        for r in reqs:
            r["spheres"] = sphere_records(r["spheres"], r["radius"])
        server = vlbm.Server(device=0, hbm_budget_bytes=16 << 30, max_resident=c["slots"])
        return dict(case=c, server=server, requests=reqs,
                    ibm=vlbm.IbmConfig.default(max_iterations=1, gx=0.0, gy=0.0, gz=-1e-5, wall_x=0, wall_y=1,
                                               wall_z=1))
    sim = vlbm.Simulation(config(c), builder=BUILDERS[c["walls"]])
    state = dict(case=c, sim=sim, n_spheres=0)
    if c["kind"] == "spheres":
        rows = sphere_set(c, seed)
        sim.init_equilibrium(1.0, *uniform_flow(seed))
        sim.add_spheres(ibm_config(c), sphere_records(rows, c["radius"]))
        state["n_spheres"] = len(rows)
    else:
        sim.set_populations(populations(c, seed).cpu().numpy())
    if c["kind"] != "report":
        shape = (c["nz"], c["ny"], c["nx"])
        state["out"] = [torch.zeros(shape, device="cuda", dtype=torch.float32) for _ in range(5)]
    torch.cuda.synchronize()
    return state


def run(state):
    c = state["case"]
    if c["kind"] == "serving":
        return run_server(state)
    sim = state["sim"]
    sim.step(c["steps"])
    if c["kind"] == "report":
        report = sim.treat_data()
        fields = sim.macroscopics()
        return dict(fields, residual=report["residual"], mean_rho=report["avg_rho"],
                    mean_uz=report["avg_uz_plane_xz"])
    rho, ux, uy, uz, omega = state["out"]
    sim.macroscopics_device(rho.data_ptr(), ux.data_ptr(), uy.data_ptr(), uz.data_ptr(), omega.data_ptr())
    out = dict(rho=rho, ux=ux, uy=uy, uz=uz, omega=omega)
    if state["n_spheres"]:
        parts = sim.particles(state["n_spheres"])
        for name in ("pos", "vel", "w"):
            out[name] = np.array([getattr(p, name)[:] for p in parts])
    return out


def run_server(state):
    server, out = state["server"], {}
    nodes = {}
    for r in state["requests"]:
        server.submit(r["cfg"], vlbm.BUILDER_DUCT_YZ, r["steps"], r["tag"], r["spheres"], state["ibm"])
        nodes[r["tag"]] = r["cfg"].nx * r["cfg"].ny * r["cfg"].nz
    while len(out) < len(nodes):
        for done in server.pump(200):
            if done.status != vlbm.OK:
                raise RuntimeError("request %d failed with status %d" % (done.tag, done.status))
            out[int(done.tag)] = server.fetch(done.tag, nodes[done.tag])
    return [out[tag] for tag in sorted(out)]


# --------------------------------------------------------------------- work --
def work(c):
    """Bytes and operations: a step reads and writes every stored population once (and the Power-Law state);
    a report reads the populations once and writes its fields; a forcing iteration reads rho and u and adds a
    force at each lattice node within reach of a sphere."""
    flops = {19: 330.0, 27: 480.0}
    if c["kind"] == "serving":
        b = f = 0.0
        for r in requests(c, 1):
            n = float(r["cfg"].nx * r["cfg"].ny * r["cfg"].nz)
            q = r["cfg"].vel_set
            b += n * (4.0 * q * r["steps"] + 4)
            f += n * flops[q] * r["steps"]
        return {"bytes": b, "flops": f}
    n, q, s = float(c["nx"] * c["ny"] * c["nz"]), c["vel_set"], 4 if c["storage"] == "f32" else 2
    per_step = 2.0 * q * s + (8 if c["rheology"] == "powerlaw" else 0)
    b = n * (per_step * c["steps"] + q * s + 20)
    f = n * flops[q] * c["steps"]
    if c["kind"] == "spheres":
        support = 4 * math.pi * c["radius"] ** 2 * 4.0   # nodes within two units of the surface
        lagrangian = 4 * math.pi * c["radius"] ** 2 * 0.76
        reps = c["spheres"] * c["steps"] * c["iterations"]
        b += reps * support * (16 + 24)
        f += reps * lagrangian * 64 * 20
    return {"bytes": b, "flops": f}


def tolerance(c):
    # Against 64 bits, single precision is off by up to 1.3e-5 (3e-5 with the Power-Law relaxation, whose
    # viscosity follows the shear rate of the step before); single values of omega vary most, near the yield
    # surface.  Half storage rounds stochastically: 2e-4 to 2e-3 off (5e-3 for omega around spheres), and another
    # implementation may take its draws in another order.
    if c["kind"] == "serving":
        return {"rel": 1e-2, "max": 0.2}
    if c["storage"] == "f32":
        return {"rel": 1e-4 if c["rheology"] == "powerlaw" else 5e-5, "max": 2e-2}
    return {"rel": 2e-2 if c["kind"] == "spheres" else 1e-2, "max": 0.5}


# -------------------------------------------------------------------- exact --
def exact(c, seed):
    if c["kind"] == "serving":
        out = []
        for r in requests(c, seed):
            if r["spheres"]:
                out.append(None)
                continue
            # from rest, periodic in x: every cross-section is alike, one is computed
            p = dict(tau=0.9, eta_p=r["cfg"].eta_p, yield_stress=r["cfg"].yield_stress, n_index=1.0, k=0.0, lid=0.0,
                     f=(r["cfg"].fx, 0.0, 0.0))
            c1 = case("fluid", None, vel_set=r["cfg"].vel_set, walls="duct", storage="f16", nx=1, ny=r["cfg"].ny,
                      nz=r["cfg"].nz, steps=r["steps"])
            ux = Exact(c1, p, rest(c1)).fields(r["steps"])["ux"]
            out.append(ux.expand(r["cfg"].nz, r["cfg"].ny, r["cfg"].nx).reshape(-1).cpu().numpy())
        return out
    e = Exact(c, physics(c), rest(c, *uniform_flow(seed)) if c["kind"] == "spheres" else populations(c, seed).double())
    if c["kind"] == "spheres":
        e.add_spheres(sphere_set(c, seed))
    out = e.fields(c["steps"])
    if c["kind"] == "spheres":
        return dict(out, pos=e.pos.cpu().numpy(), vel=e.vel.cpu().numpy(), w=e.w.cpu().numpy())
    if c["kind"] == "report":
        # the residual of a first report is taken against fluid at rest
        return dict({k: v.cpu().numpy() for k, v in out.items()}, residual=1.0, mean_rho=float(out["rho"].mean()),
                    mean_uz=out["uz"].mean(dim=(0, 2)).cpu().numpy())
    return out


def rest(c, ux=0.0, uy=0.0, uz=0.0):
    f = torch.empty((c["vel_set"], c["nz"], c["ny"], c["nx"]), device=device(), dtype=torch.float64)
    ux, uy, uz = (float(np.float32(v)) for v in (ux, uy, uz))
    for i, (cx, cy, cz) in enumerate(C27[:c["vel_set"]]):
        cu = cx * ux + cy * uy + cz * uz
        f[i] = weight(c["vel_set"], i) * (1 - 1.5 * (ux * ux + uy * uy + uz * uz) + 3 * cu + 4.5 * cu * cu)
    return f


class Exact:
    """The time step in 64 bits: push streaming into a second array, boundary rules on the streamed values."""

    def __init__(self, c, p, f):
        self.c, self.p, self.f, self.q = c, p, f, c["vel_set"]
        self.shape = tuple(f.shape[1:])
        self.eta, self.first, self.force, self.spheres = None, True, None, False

    def moments(self, f, force):
        rho, j, s = f.sum(0), [0.0] * 3, {}
        for i in range(1, self.q):
            ci = C27[i]
            for a in range(3):
                if ci[a]:
                    j[a] = j[a] + ci[a] * f[i]
                for b in range(a, 3):
                    if ci[a] * ci[b]:
                        s[a, b] = s.get((a, b), 0.0) + ci[a] * ci[b] * f[i]
        u = [(j[a] + 0.5 * force[a]) / rho for a in range(3)]
        for a, b in s:
            s[a, b] = s[a, b] - rho * u[a] * u[b] - (rho / 3 if a == b else 0)
        return rho, u, s

    def omega(self, u, pi, force):
        p, kind = self.p, self.c["rheology"]
        if kind == "newtonian":
            return torch.full(self.shape, 1 / p["tau"], device=self.f.device, dtype=torch.float64), None
        total = 0.0
        for a in range(3):
            for b in range(a, 3):
                t = pi[a, b] + 0.5 * (u[a] * force[b] + u[b] * force[a])
                total = total + (1 if a == b else 2) * t * t
        size = torch.sqrt(0.5 * total)
        if kind == "bingham":
            return (1 / (3 * p["eta_p"] + 0.5)) * torch.clamp(1 - p["yield_stress"] / size, min=0.0), None
        # the shear rate follows from the stress and the previous step's apparent viscosity
        gamma = 3 * size / (0.5 + 3 * self.eta) if self.eta is not None else torch.zeros_like(size)
        eta = torch.where(gamma <= 0, torch.full_like(gamma, p["k"]), p["k"] * gamma.clamp(min=1e-300) ** (p["n_index"] - 1))
        return 1 / (0.5 + 3 * eta), eta

    def step(self):
        f, q = self.f, self.q
        force = list(self.p["f"])
        if self.force is not None:
            force = [force[a] + self.force[a] for a in range(3)]
        rho, u, pi = self.moments(f, force)
        omega, self.eta = self.omega(u, pi, force)
        half = 1 - 0.5 * omega
        uu = sum(v * v for v in u)
        uf = sum(v * g for v, g in zip(u, force))
        trace = (pi[0, 0] + pi[1, 1] + pi[2, 2]) / 3
        after = torch.empty_like(f)
        for i in range(q):
            ci, w = C27[i], weight(q, i)
            cu, cf = (sum(ci[a] * v[a] for a in range(3)) for v in (u, force))
            eq = rho * (1 - 1.5 * uu + 3 * cu + 4.5 * cu * cu)
            push = half * (3 * (cf - uf) + 9 * cu * cf)
            if self.c["operator"] == "bgk":
                after[i] = (1 - omega) * f[i] + w * (omega * eq + push)
            else:
                qp = -trace
                for a in range(3):
                    for b in range(a, 3):
                        if ci[a] * ci[b]:
                            qp = qp + (1 if a == b else 2) * ci[a] * ci[b] * pi[a, b]
                after[i] = w * (4.5 * (1 - omega) * (qp - cf / 3) + eq + push)
        new = f   # its values are no longer needed
        for i in range(q):
            cx, cy, cz = C27[i]
            new[i] = torch.roll(after[i], (cz, cy, cx), (0, 1, 2))
        self.walls(new, after)
        self.f = new
        self.force = None
        if self.spheres:
            self.immersed()

    def walls(self, new, after):
        q, wall = self.q, WALLS[self.c["walls"]]
        sides = [(-1, 0, 1) if w else (0,) for w in wall]
        for sx in sides[0]:
            for sy in sides[1]:
                for sz in sides[2]:
                    side = (sx, sy, sz)
                    if side == (0, 0, 0):
                        continue
                    where = []
                    for a, n in zip((2, 1, 0), self.shape):
                        where.append(slice(None) if not wall[a] else slice(0, 1) if side[a] < 0 else
                                     slice(n - 1, n) if side[a] > 0 else slice(1, n - 1))
                    where = tuple(where)
                    lid = self.c["walls"] == "cavity" and side == (0, 1, 0)
                    density = new[(slice(None),) + where].sum(0) if lid else None
                    for i in range(1, q):
                        d = [C27[i][a] * side[a] for a in range(3)]
                        if not (min(d) < 0 <= max(d) and max(d) <= 0):   # comes from a wall, crosses none outward
                            continue
                        o = i + 1 if i % 2 else i - 1
                        if lid:
                            speed = C27[o][0] * float(np.float32(self.p["lid"]))
                            new[(i,) + where] = new[(o,) + where] - 6 * density * weight(q, i) * speed
                        else:
                            new[(i,) + where] = after[(o,) + where]

    def fields(self, steps):
        for _ in range(steps):
            self.step()
        force = list(self.p["f"])
        rho, u, pi = self.moments(self.f, force)
        omega, _ = self.omega(u, pi, force)
        if self.spheres:   # what the forcing left at the nodes that it reached
            rho, u = self.rho, self.u
        return dict(rho=rho, ux=u[0], uy=u[1], uz=u[2], omega=omega)

    # spheres: Lagrangian nodes on each surface, Peskin's four-point kernel, direct forcing
    def add_spheres(self, rows):
        r, dev = self.c["radius"], self.f.device
        x, area = surface(r)
        t = lambda v: torch.tensor(v, device=dev, dtype=torch.float64)  # noqa: E731
        rows = t(rows)
        self.pos, self.vel, self.w = rows[:, 0:3].clone(), rows[:, 3:6].clone(), rows[:, 6:9].clone()
        self.nodes = (self.pos[:, None, :] + t(x)[None]).reshape(-1, 3)
        self.area, self.of = t(area).repeat(len(rows)), torch.arange(len(rows), device=dev).repeat_interleave(len(area))
        self.last_force = torch.zeros_like(self.pos)
        self.length = t([float(self.c["nx"]), float(self.c["ny"]), float(self.c["nz"])])
        self.walled = torch.tensor([bool(w) for w in WALLS[self.c["walls"]]], device=dev)
        self.spheres = True

    def near(self, d):
        """The nearest image of a difference on the periodic axes."""
        return torch.where(self.walled, d, d - self.length * torch.round(d / self.length))

    def immersed(self):
        c, dev = self.c, self.f.device
        force = self.p["f"]
        rho, u, _ = self.moments(self.f, force)
        u = [v.reshape(-1).clone() for v in u]
        flat = rho.reshape(-1)
        volume, density = c["radius"] ** 3 * 4 * math.pi / 3, 1.5
        inertia = 2.0 * volume * density * c["radius"] ** 2 / 5.0
        old_pos, old_vel, old_w, old_force = self.pos, self.vel, self.w, self.last_force
        gravity = torch.tensor([0.0, 0.0, -1e-5], device=dev, dtype=torch.float64)

        def centre(f, m):
            self.vel = old_vel + ((0.5 * old_force + 0.5 * f) / volume + (density - 1.0) * gravity) / density
            self.w = old_w + 0.5 * m / inertia

        f, m = torch.zeros_like(self.pos), torch.zeros_like(self.pos)
        centre(f, m)
        base = torch.trunc(self.nodes) - 1
        k = torch.arange(4, device=dev, dtype=torch.float64)
        r = (k - (self.nodes - base)[:, :, None]).abs()
        weights = torch.where(r <= 1, (3 - 2 * r + torch.sqrt((1 + 4 * r - 4 * r * r).clamp(min=0))) / 8,
                              torch.where(r <= 2, (5 - 2 * r - torch.sqrt((-7 + 12 * r - 4 * r * r).clamp(min=0))) / 8,
                                          torch.zeros_like(r)))
        at = (base[:, :, None] + k).to(torch.int64)                       # [node][axis][4]
        size = torch.tensor([c["nx"], c["ny"], c["nz"]], device=dev)[None, :, None]
        inside = ~self.walled[None, :, None] | ((at >= 0) & (at < size))
        weights = weights * inside
        at = at % size
        index = (at[:, 2, :, None, None] * c["ny"] + at[:, 1, None, :, None]) * c["nx"] + at[:, 0, None, None, :]
        delta = weights[:, 2, :, None, None] * weights[:, 1, None, :, None] * weights[:, 0, None, None, :]
        index, delta = index.reshape(len(index), 64), delta.reshape(len(delta), 64)
        arm = self.near(self.nodes - self.pos[self.of])
        added = [torch.zeros_like(flat) for _ in range(3)]
        for _ in range(c["iterations"]):
            local = (flat[index] * delta).sum(1)
            speed = torch.stack([(v[index] * delta).sum(1) for v in u], 1)
            wanted = self.vel[self.of] + torch.linalg.cross(self.w[self.of], arm)
            df = (2 * local * self.area)[:, None] * (speed - wanted)
            f = f.index_add(0, self.of, df)
            m = m.index_add(0, self.of, torch.linalg.cross(arm, df))
            centre(f, m)
            for a in range(3):
                spread = torch.zeros_like(flat).index_add_(0, index.reshape(-1), (-df[:, a, None] * delta).reshape(-1))
                u[a] += 0.5 * spread / flat
                added[a] += spread
        self.last_force = f
        wrap = lambda x: torch.where(self.walled, x, torch.fmod(x + self.length, self.length))  # noqa: E731
        self.pos = wrap(old_pos + 0.5 * (self.vel + old_vel))
        # nodes turn with the sphere's mean rotation about its old centre
        avg = (0.5 * (self.w + old_w))[self.of]
        size = torch.linalg.norm(avg, dim=1)
        v = self.near(self.nodes - old_pos[self.of])
        q0 = torch.cos(0.5 * size)
        qv = avg / size[:, None].clamp(min=1e-300) * torch.sin(0.5 * size)[:, None]
        t, (qi, qj, qk) = q0 * q0 - 0.5, qv.unbind(1)
        # the third row as the reference program has it (qi qj - q0 qj)
        turned = 2 * torch.stack([(t + qi * qi) * v[:, 0] + (qi * qj - q0 * qk) * v[:, 1] + (qi * qk + q0 * qj) * v[:, 2],
                                  (qi * qj + q0 * qk) * v[:, 0] + (t + qj * qj) * v[:, 1] + (qj * qk - q0 * qi) * v[:, 2],
                                  (qi * qj - q0 * qj) * v[:, 0] + (qj * qk + q0 * qi) * v[:, 1] + (t + qk * qk) * v[:, 2]], 1)
        moved = torch.where((size > 1e-8)[:, None], self.pos[self.of] + turned,
                            self.nodes + self.near(self.pos - old_pos)[self.of])
        self.nodes = wrap(moved)
        self.rho, self.u = rho, [v.reshape(self.shape) for v in u]
        self.force = [v.reshape(self.shape) for v in added]


def surface(r):
    """Lagrangian nodes of a sphere about its centre, in layers, and the area of each (unit mesh scale)."""
    layers = int(2.0 * math.sqrt(2.0) * r + 1.0)
    theta = [math.pi * (i / layers - 0.5) for i in range(layers + 1)]
    count = [int(1.5 + math.cos(t) * layers * math.sqrt(3.0)) for t in theta]
    zeta = [r * math.sin(t) for t in theta]
    cap = [(zeta[i] + zeta[i + 1]) / 2.0 - zeta[0] for i in range(layers)] + [2 * r]
    cap = [2 * math.pi * r * v for v in cap]
    ring = [cap[0]] + [cap[i] - cap[i - 1] for i in range(1, layers + 1)]
    ring[0] = ring[layers]
    x, area, phase = [(0.0, 0.0, zeta[0])], [ring[0]], 0.0
    for i in range(1, layers):
        if i % 2:
            phase += math.pi / count[i]
        for j in range(count[i]):
            a = j * 2.0 * math.pi / count[i] + phase
            x.append((r * math.cos(theta[i]) * math.cos(a), r * math.cos(theta[i]) * math.sin(a), zeta[i]))
            area.append(ring[i] / count[i])
    x.append((0.0, 0.0, zeta[layers]))
    area.append(ring[layers])
    return x, area
