"""The workloads this library is timed on: what a case is, how its state is made,
one pass of it through the public entry points, and its result in 64 bits.

A case is a dict of plain values; `kind` says which program it stands for:

  thread    one periodic (or wetting-walled) domain stepped by Lattice.step,
            its fields read back every `steps` steps (a parameter study's run)
  sphere    the same with one moving sphere between wetting walls
  reference the reference's own geometry and 12 particles, stepped whole
  driver    the same, one library call per subroutine, as a Fortran driver does
  batch     many uneven domains stepped together, half of them with a sphere
  exchange  a host program that uploads populations, steps, downloads them
  serve     jobs submitted to the server and run to their step limit

Fields come back in the precision of the storage the program chose: 64 bits
for FP64, 32 for FP32 and 16 for the 16-bit storage, as its snapshots keep them.
"""
import math

import numpy as np
import torch

from symmetry_b200 import configs
from symmetry_b200.lib import Batch, Lattice, Server, job_spec
from symmetry_b200.params import SymParticles, config_params, particles_get, particles_set, reference_params

FIELDS = ("rho", "ux", "uy", "uz", "rho_N")
KEPT = {"fp64": torch.float64, "fp32": torch.float32, "fp16": torch.float16}
POP_BYTES = {"fp64": 8, "fp32": 4, "fp16": 2}
PHI_BYTES = {"fp64": 8, "fp32": 4, "fp16": 4}
# the loop body of the reference's main, one entry point per subroutine
DRIVER = ("calmacros", "lagrange_points", "capillary_force2", "momentum", "repulsive", "movement", "set_walls",
          "refilling", "derivatives", "collision", "recolor", "boundary", 0, 1, "curve")


def listed():
    return [
        # the smallest domain of the configurations: launches and latency
        dict(name="thread_32x32x96_fp64", kind="thread", storage="fp64", nx=32, ny=32, nz=96, steps=10, wall=0),
        # a domain of the batched mix stepped by itself, no extent a multiple of a tile
        dict(name="thread_53x53x374_fp64", kind="thread", storage="fp64", nx=53, ny=53, nz=374, steps=20, wall=0),
        # the precision study's thread at its full size: the largest
        dict(name="thread_256x256x512_fp64", kind="thread", storage="fp64", nx=256, ny=256, nz=512, steps=50, wall=0),
        # the study's half-size thread in FP32, between wetting walls as 30 % of served jobs have them
        dict(name="wall_128x128x256_fp32", kind="thread", storage="fp32", nx=128, ny=128, nz=256, steps=100, wall=1),
        # the large served thread in 16-bit storage
        dict(name="thread_128x128x512_fp16", kind="thread", storage="fp16", nx=128, ny=128, nz=512, steps=100,
             wall=0),
        # wetting walls and one moving sphere, the second configuration
        dict(name="sphere_64x64x128_fp64", kind="sphere", storage="fp64", nx=64, ny=64, nz=128, steps=20, rad=8.0),
        # the reference program as written: 152^3, 12 particles
        dict(name="reference_152x152x152", kind="reference", nx=152, ny=152, nz=152, steps=20),
        # a Fortran driver calling one subroutine after another, at the parity tests' size
        dict(name="driver_48x88x48", kind="driver", nx=48, ny=88, nz=48, steps=4),
        # the batched mix, a quarter of it, in 16-bit storage
        dict(name="batch_24_fp16", kind="batch", storage="fp16", domains=24, mix=4, lo=24, hi=64, steps=100),
        # a few small uneven domains in FP32
        dict(name="batch_6_fp32", kind="batch", storage="fp32", domains=6, mix=9, lo=16, hi=33, steps=50),
        # populations from the host and back, ten steps between (a coupled host program, a restart)
        dict(name="exchange_64x64x128_fp64", kind="exchange", storage="fp64", nx=64, ny=64, nz=128, steps=10),
        # five served jobs of the batched mix's sizes run to a step limit
        dict(name="serve_5_fp16", kind="serve", storage="fp16", jobs=5, mix=5, lo=24, hi=64, steps=200),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["thread", "thread", "thread", "sphere", "reference", "driver", "batch", "exchange", "serve"])
    storage = rng.choice(["fp64", "fp32", "fp16"])
    if kind == "thread":
        # to the largest listed size in FP64; reduced storage to the served size
        big = storage == "fp64"
        nx, nz = _log(rng, 16, 200 if big else 128), _log(rng, 32, 512)
        ny = max(16, min(200 if big else 128, nx + rng.randint(-9, 9)))
        return dict(kind=kind, storage=storage, nx=nx, ny=ny, nz=nz, steps=rng.randint(10, 50), wall=rng.randint(0, 1))
    if kind == "sphere":
        n = _log(rng, 32, 96)
        return dict(kind=kind, storage=storage, nx=n, ny=n + rng.randint(-3, 3), nz=_log(rng, 64, 192),
                    steps=rng.randint(10, 40), rad=float(rng.randint(4, 8)))
    if kind in ("reference", "driver"):
        hi = 160 if kind == "reference" else 96
        return dict(kind=kind, nx=_log(rng, 48, hi), ny=_log(rng, 88, hi), nz=_log(rng, 48, hi),
                    steps=rng.randint(2, 10))
    if kind == "batch":
        return dict(kind=kind, storage=storage, domains=rng.randint(3, 20), mix=rng.randint(0, 9999),
                    lo=rng.choice([16, 24]), hi=rng.choice([32, 64]), steps=rng.randint(10, 60))
    if kind == "exchange":
        n = _log(rng, 20, 80)
        return dict(kind=kind, storage=storage, nx=n, ny=n + rng.randint(-4, 4), nz=_log(rng, 40, 160),
                    steps=rng.randint(1, 20))
    return dict(kind=kind, storage=storage, jobs=rng.randint(2, 6), mix=rng.randint(0, 9999), lo=24,
                hi=rng.choice([32, 64]), steps=rng.randint(50, 200))


# ---- domains --------------------------------------------------------------------
def _domains(case):
    """The single domains of a case: (params, red radius or slab, wavelength, sphere)."""
    kind = case["kind"]
    if kind in ("thread", "exchange"):
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        p = config_params(nx, ny, nz, tau_r=0.8, sigma=5e-3, storage=case["storage"], wall_x=bool(case.get("wall")),
                          cita_deg=60.0 if case.get("wall") else 90.0)
        return [dict(p=p, radius=0.2 * min(nx, ny), wavelength=float(nz))]
    if kind == "sphere":
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        p = config_params(nx, ny, nz, tau_r=0.8, sigma=5e-3, wall_x=True, cita_deg=60.0, par=1, rad=case["rad"],
                          rho_p_ratio=1.5, body=(0.0, 0.0, -1e-6), storage=case["storage"])
        return [dict(p=p, slab=(0.3 * nz, 0.7 * nz), centre=(nx / 2.0, ny / 2.0, 0.3 * nz))]
    # batch, serve: the batched mix's distribution of sizes, viscosities and tensions
    rng = np.random.default_rng(case["mix"])
    out = []
    for k in range(case["domains"] if kind == "batch" else case["jobs"]):
        n = int(rng.integers(case["lo"], case["hi"] + 1))
        radius = float(rng.uniform(4.0, 0.3 * n))
        lam = float(rng.uniform(0.7, 2.0)) * 2.0 * math.pi * radius
        nwave = max(1, int(round(rng.integers(2 * case["lo"], 6 * case["hi"] + 1) / lam)))
        nz = max(16, int(round(nwave * lam)))
        sphere = k % 2 == 1
        p = config_params(n, n, nz, tau_r=float(rng.uniform(0.8, 1.5)), sigma=float(rng.uniform(2e-3, 1e-2)),
                          par=1 if sphere else 0, rad=max(3.0, radius / 2.0) if sphere else 0.0, rho_p_ratio=1.2,
                          storage=case["storage"])
        d = dict(p=p, radius=radius, wavelength=nz / nwave)
        if sphere:
            d["centre"] = ((n - 1) / 2.0, (n - 1) / 2.0, nz / 2.0)
        out.append(d)
    return out


def _start(d, seed):
    """Phase field, density and velocity a program starts domain `d` from: a
    perturbed thread (or slab) with seed noise, in a background shear flow."""
    p = d["p"]
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    a = torch.rand(4, generator=gen, device="cuda", dtype=torch.float64)
    x, y, z = (torch.arange(n, device="cuda", dtype=torch.float64) for n in (p.nx, p.ny, p.nz))
    x, y, z = x[:, None, None], y[None, :, None], z[None, None, :]
    tau = 2.0 * math.pi
    if "slab" in d:
        z0, z1 = d["slab"]
        phi = torch.tanh(torch.minimum(z - z0, z1 - z)).expand(p.nx, p.ny, p.nz)
        jump = 0.0
    else:
        rz = d["radius"] * (1.0 + 0.05 * torch.cos(tau * (z / d["wavelength"] + a[0])))
        phi = torch.tanh(rz - torch.sqrt((x - (p.nx - 1) / 2.0) ** 2 + (y - (p.ny - 1) / 2.0) ** 2))
        jump = 3.0 * p.sigma / rz
    noise = torch.rand(p.nx, p.ny, p.nz, generator=gen, device="cuda", dtype=torch.float64)
    phi = (phi + 1e-4 * (2.0 * noise - 1.0)).clamp(-1.0, 1.0)
    rho = p.rho0 + torch.where(phi > 0, phi * 0 + jump, phi * 0)
    one = torch.ones_like(phi)
    u = torch.stack([0.02 * torch.sin(tau * (y / p.ny + a[1])) * one, 0.02 * torch.sin(tau * (z / p.nz + a[2])) * one,
                     0.03 + 0.02 * torch.sin(tau * (x / p.nx + a[3])) * one])
    return phi, rho, u


def _equilibrium(rho, u):
    """Second-order equilibrium populations, velocity index first."""
    c = torch.tensor(C, device=rho.device, dtype=rho.dtype)
    w = torch.tensor(W, device=rho.device, dtype=rho.dtype)
    usq = (u * u).sum(0)
    out = torch.empty((19,) + tuple(rho.shape), device=rho.device, dtype=rho.dtype)
    for i in range(19):
        uc = c[i, 0] * u[0] + c[i, 1] * u[1] + c[i, 2] * u[2]
        out[i] = w[i] * rho * (1 + 3 * uc + 4.5 * uc * uc - 1.5 * usq)
    return out


def _host(pops):
    """Populations (19, x, y, z) on the device -> the host layout (x, y, z, 19)."""
    return pops.movedim(0, -1).contiguous().cpu().numpy()


def _lattice(d, seed):
    """A domain set up by its program: masks, then the populations it starts from."""
    p = d["p"]
    lat = Lattice(p)
    if p.par:
        s = SymParticles()
        particles_set(s, "center", 1, [d["centre"]])
        particles_set(s, "center0", 1, [d["centre"]])
        particles_set(s, "up", 1, [(0.0, 0.0, 0.03)])
        lat.set_particles(s)
    lat.call("set_walls")
    phi, rho, u = _start(d, seed)
    if p.storage == 0 and not p.par:
        # FP64 domains start at rest, from the phase field and the density
        lat.init_phase(phi.cpu().numpy(), rho.cpu().numpy())
    else:
        red = rho * (1.0 + phi) / 2.0
        lat.set_populations(_host(_equilibrium(red, u)), _host(_equilibrium(rho - red, u)))
        lat.set("rho_N", phi.cpu().numpy())
    lat.call("derivatives")
    return lat


class _Fields:
    """Pinned arrays the fields of some domains are read into, one per field."""

    def __init__(self, lattices, kept):
        n = sum(lat.p.n_nodes for lat in lattices)
        self.flat = {k: torch.empty(n, dtype=torch.float64, pin_memory=True) for k in FIELDS}
        self.kept = None if kept == torch.float64 else {k: torch.empty(n, dtype=kept) for k in FIELDS}
        self.parts, at = [], 0
        for lat in lattices:
            m = lat.p.n_nodes
            self.parts.append((lat, {k: v[at:at + m].numpy() for k, v in self.flat.items()}))
            at += m

    def read(self):
        for lat, out in self.parts:
            lat.macros(out)
        if self.kept is None:
            return self.flat
        for k in FIELDS:
            self.kept[k].copy_(self.flat[k])
        return self.kept


def _motion(lat):
    s = lat.particles()
    return {k: np.array(particles_get(s, k, lat.p.par)) for k in ("center", "up", "rp")}


# ---- the state a program holds, and one pass ---------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind in ("reference", "driver"):
        p = reference_params(case["nx"], case["ny"], case["nz"])
        lat = Lattice(p)
        lat.initia_center()
        lat.call("set_walls")
        lat.initialization()
        # another seed is another thread: the phase field with its own noise
        gen = torch.Generator(device="cuda").manual_seed(int(seed))
        noise = torch.rand(lat.shape, generator=gen, device="cuda", dtype=torch.float64)
        phi = (torch.from_numpy(lat.get("rho_N")).cuda() + 1e-4 * (2.0 * noise - 1.0)).clamp(-1.0, 1.0)
        lat.init_phase(phi.cpu().numpy(), lat.get("rho"))
        lat.call("derivatives")
        return dict(case=case, lat=lat, out=_Fields([lat], torch.float64))
    if kind == "serve":
        specs = []
        for k, d in enumerate(_domains(case)):
            gen = dict(radius=d["radius"], amp=0.05, wavelength=d["wavelength"], seed=int(seed) * 64 + k)
            parts = [dict(center=list(d["centre"]))] if "centre" in d else []
            specs.append(job_spec(configs.Workload("job%d" % k, d["p"], "thread", gen, case["steps"], parts),
                                  case["steps"] - 10 * k))
        return dict(case=case, server=Server(), specs=specs)
    ds = _domains(case)
    lats = [_lattice(d, int(seed) * 64 + k) for k, d in enumerate(ds)]
    kept = KEPT[case["storage"]]
    if kind == "exchange":
        phi, rho, u = _start(ds[0], int(seed) * 64)
        red = rho * (1.0 + phi) / 2.0
        pops = [torch.from_numpy(_host(_equilibrium(v, u))).pin_memory() for v in (red, rho - red)]
        back = [torch.empty(v.shape, dtype=v.dtype, pin_memory=True) for v in pops]
        return dict(case=case, lat=lats[0], pops=pops, back=back,
                    kept=None if kept == torch.float64 else [torch.empty(v.shape, dtype=kept) for v in back])
    if kind == "batch":
        free = [lat for lat in lats if not lat.p.par]
        held = [lat for lat in lats if lat.p.par]
        return dict(case=case, batch=Batch(lats), held=held, out=[_Fields(free, kept), _Fields(held, kept)])
    return dict(case=case, lat=lats[0], out=_Fields(lats, kept))


def run(state):
    case = state["case"]
    kind, steps = case["kind"], case["steps"]
    if kind == "serve":
        server = state["server"]
        ids = [server.submit(s) for s in state["specs"]]
        server.run_until_idle()
        done = [server.result(i) for i in ids]
        return dict(rmin=np.array([r.rmin for r in done], dtype=np.float32),
                    steps=np.array([r.steps for r in done], dtype=np.int32))
    if kind == "batch":
        state["batch"].step(steps)
        return dict(free=state["out"][0].read(), held=state["out"][1].read(),
                    motion=[_motion(lat) for lat in state["held"]] if case["storage"] == "fp64" else None)
    lat = state["lat"]
    if kind == "exchange":
        lat.set_populations(state["pops"][0].numpy(), state["pops"][1].numpy())
        lat.step(steps)
        for name, back in zip(("ri", "bi"), state["back"]):
            lat.get_into(name, back.numpy())
        if state["kept"] is None:
            return state["back"]
        for kept, back in zip(state["kept"], state["back"]):
            kept.copy_(back)
        return state["kept"]
    if kind == "driver":
        for _ in range(steps):
            for sub in DRIVER:
                if isinstance(sub, int):
                    lat.streaming(sub)
                else:
                    lat.call(sub)
    else:
        lat.step(steps)
    fields = state["out"].read()
    if kind == "thread":
        return fields
    return dict(fields=fields, motion=_motion(lat) if case.get("storage", "fp64") == "fp64" else None)


def work(case):
    kind, steps = case["kind"], case["steps"]
    if kind in ("reference", "driver"):
        ps, nodes = "fp64", [case["nx"] * case["ny"] * case["nz"]]
    else:
        ps, nodes = case["storage"], [d["p"].n_nodes for d in _domains(case)]
    # a step reads and writes 38 populations a node, writes the phase field and reads it
    step = 76 * POP_BYTES[ps] + 2 * PHI_BYTES[ps]
    if kind == "serve":
        every = [n * (steps - 10 * k) for k, n in enumerate(nodes)]
        return dict(bytes=step * sum(every), flops=600 * sum(every))
    n = sum(nodes)
    # the fields (or populations) that cross between host and device
    moved = 4 * 19 * 8 if kind == "exchange" else 5 * 8
    return dict(bytes=n * (step * steps + moved), flops=600 * n * steps)


# ---- the same in 64 bits, from the model's definition ---------------------------------
C = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 0), (-1, 1, 0),
     (1, -1, 0), (-1, -1, 0), (1, 0, 1), (-1, 0, 1), (1, 0, -1), (-1, 0, -1), (0, 1, 1), (0, -1, 1), (0, 1, -1),
     (0, -1, -1)]
W = [1 / 3 if sum(map(abs, c)) == 0 else 1 / 18 if sum(map(abs, c)) == 1 else 1 / 36 for c in C]


def _moments():
    rows = []
    for x, y, z in C:
        s = x * x + y * y + z * z
        rows.append([1, 19 * s - 30, (21 * s * s - 53 * s + 24) / 2, x, (5 * s - 9) * x, y, (5 * s - 9) * y, z,
                     (5 * s - 9) * z, 3 * x * x - s, (3 * s - 5) * (3 * x * x - s), y * y - z * z,
                     (3 * s - 5) * (y * y - z * z), x * y, y * z, x * z, (y * y - z * z) * x, (z * z - x * x) * y,
                     (x * x - y * y) * z])
    m = torch.tensor(rows, dtype=torch.float64).T.contiguous()
    return m, (m / (m * m).sum(1, keepdim=True)).T.contiguous()


class _Exact:
    """The lattice update in 64 bits: periodic box, optional wetting wall planes
    at both ends of x, no particles."""

    def __init__(self, d, seed, at_rest):
        self.p = p = d["p"]
        phi, rho, u = _start(d, seed)
        red = rho * (1.0 + phi) / 2.0
        u = torch.zeros_like(u) if at_rest else u
        self.f = torch.stack([_equilibrium(red, u), _equilibrium(rho - red, u)])   # colour, velocity, node
        self.m, self.minv = (v.cuda() for v in _moments())
        solid = torch.zeros_like(phi, dtype=torch.bool)
        self.wall = torch.zeros_like(phi)   # inward x normal of the wall a node belongs to
        if p.wall_x:
            solid[0] = solid[-1] = True
            self.wall[0], self.wall[-1] = 1.0, -1.0
        self.solid = solid
        self.near = torch.zeros_like(phi)   # fluid next to a wall: that wall's normal
        for c in C[1:]:
            nb = self.at(self.wall, c)
            self.near = torch.where(~solid & (nb != 0), nb, self.near)

    @staticmethod
    def at(v, c):
        """v at node x + c"""
        dims = [k for k in range(3) if c[k]]
        return torch.roll(v, [-c[k] for k in dims], [k - 3 for k in dims]) if dims else v

    def macros(self):
        """density, velocity and phase field of the populations; red, blue, total populations"""
        red, blue = self.f[0].sum(0), self.f[1].sum(0)
        tot = self.f[0] + self.f[1]
        rho = red + blue
        mom = [sum(c[k] * tot[i] for i, c in enumerate(C) if c[k]) for k in range(3)]
        zero = torch.zeros_like(rho)
        u = torch.stack([torch.where(self.solid, zero, v / rho) for v in mom])
        phi = torch.where(self.solid, zero, (red - blue) / rho)
        return torch.where(self.solid, zero + self.p.rho0, rho), u, phi, red, blue, tot

    def step(self):
        p, solid, walls = self.p, self.solid, bool(self.p.wall_x)
        rho, u, phi, red, blue, tot = self.macros()
        zero = torch.zeros_like(rho)
        if walls:   # a wall node's phase field: the weighted mean of its fluid neighbours
            ws, v = zero.clone(), zero.clone()
            for w, c in zip(W[1:], C[1:]):
                fluid = (~self.at(solid, c)).to(phi.dtype)
                ws += w * fluid
                v += w * fluid * self.at(phi, c)
            phi = torch.where(solid & (ws > 0), v / ws.clamp_min(1e-300), phi)
        g = torch.zeros_like(u)
        for w, c in zip(W[1:], C[1:]):
            nb = self.at(phi, c)
            for k in range(3):
                if c[k]:
                    g[k] += 3.0 * w * c[k] * nb
        norm = (g * g).sum(0).sqrt()
        flag = (norm > p.evap_lim) & ~solid
        n = torch.where(flag, g / norm.clamp_min(1e-300), torch.zeros_like(g))
        g = torch.where(solid, torch.zeros_like(g), g)
        if walls:   # rotated to the contact angle next to a wall
            wet = flag & (self.near != 0)
            nw = torch.stack([self.near, zero, zero])
            th = torch.where((nw - n).abs().amax(0) < 1e-5, zero + 1e-5, torch.acos((nw * n).sum(0).clamp(-1, 1)))
            s, co = math.sin(p.cita), math.cos(p.cita)
            v1 = (co - s * th.cos() / th.sin()) * nw + s / th.sin() * n
            v2 = (co + s * th.cos() / th.sin()) * nw - s / th.sin() * n
            rot = torch.where(((v1 - n) ** 2).sum(0) < ((v2 - n) ** 2).sum(0), v1, v2)
            n = torch.where(wet, rot, n)
            g = torch.where(wet, norm * rot, g)
        d = [[zero.clone() for _ in range(3)] for _ in range(3)]
        for w, c in zip(W[1:], C[1:]):
            nb = self.at(n, c)
            for a in range(3):
                for b in range(3):
                    if c[b]:
                        d[a][b] += 3.0 * w * c[b] * nb[a]
        kurv = (n[0] * n[1] * (d[1][0] + d[0][1]) + n[0] * n[2] * (d[2][0] + d[0][2]) +
                n[1] * n[2] * (d[1][2] + d[2][1]) - (n[1] ** 2 + n[2] ** 2) * d[0][0] -
                (n[0] ** 2 + n[2] ** 2) * d[1][1] - (n[0] ** 2 + n[1] ** 2) * d[2][2])
        force = torch.where(flag & (self.near == 0), 0.5 * p.sigma * kurv * g, torch.zeros_like(g))
        u = u + 0.5 * force / rho
        ph = phi.clamp(-1.0, 1.0)
        nu = 2.0 / ((1 + ph) / p.nu_r + (1 - ph) / p.nu_b)
        su = 1.0 / (3.0 * nu + 0.5)
        sq = 8.0 * (2.0 - su) / (8.0 - su)
        one = torch.ones_like(su)
        rate = torch.stack([one, su, su, one, sq, one, sq, one, sq, su, su, su, su, su, su, su, sq, sq, sq])
        ux, uy, uz = u
        fx, fy, fz = force
        usq, uf = (u * u).sum(0), (u * force).sum(0)
        eq = rho * torch.stack([one, 19 * usq - 11, 3 - 5.5 * usq, ux, -ux / 1.5, uy, -uy / 1.5, uz, -uz / 1.5,
                                3 * ux * ux - usq, -0.5 * (3 * ux * ux - usq), uy * uy - uz * uz,
                                -0.5 * (uy * uy - uz * uz), ux * uy, uy * uz, ux * uz, zero, zero, zero])
        fk = torch.stack([zero, 38 * uf, -11 * uf, fx, -fx / 1.5, fy, -fy / 1.5, fz, -fz / 1.5, 6 * ux * fx - 2 * uf,
                          uf - 3 * ux * fx, 2 * (uy * fy - uz * fz), uz * fz - uy * fy, ux * fy + uy * fx,
                          uy * fz + uz * fy, ux * fz + uz * fx, zero, zero, zero])
        m = torch.tensordot(self.m, tot, 1)
        m = m - rate * (m - eq) + (1.0 - 0.5 * rate) * fk
        post = torch.tensordot(self.minv, m, 1)
        share, mix = red / rho, torch.where(flag, red * blue / rho * p.beta, zero)
        new = torch.empty_like(self.f)
        for i, (w, c) in enumerate(zip(W, C)):
            r = share * post[i] + (mix * w * (c[0] * n[0] + c[1] * n[1] + c[2] * n[2]) if i else 0.0)
            r = torch.where(red <= p.evap_lim, zero, r)
            r = torch.where(blue <= p.evap_lim, post[i], r)
            new[0, i], new[1, i] = r, post[i] - r
        if walls:
            new = torch.where(solid, self.f, new)
        out = torch.empty_like(new)
        for i, c in enumerate(C):
            back = tuple(-v for v in c)
            out[:, i] = self.at(new[:, i], back)
            if walls and i:   # what comes out of a wall is what went in
                came = self.at(solid, back) & ~solid
                out[:, i] = torch.where(came, new[:, C.index(back)], out[:, i])
        self.f = out


def exact(case, seed):
    kind = case["kind"]
    if kind not in ("thread", "batch", "exchange"):
        return None
    at_rest = case["storage"] == "fp64" and kind != "exchange"
    if kind == "exchange" or kind == "thread":
        e = _Exact(_domains(case)[0], int(seed) * 64, at_rest)
        for _ in range(case["steps"]):
            e.step()
        if kind == "exchange":
            return [e.f[k].movedim(0, -1).cpu() for k in range(2)]
        rho, u, phi = e.macros()[:3]
        return {k: v.reshape(-1).cpu() for k, v in zip(FIELDS, (rho, u[0], u[1], u[2], phi))}
    if case["domains"] * case["steps"] > 3000:
        return None
    got = {k: [] for k in FIELDS}
    for k, d in enumerate(_domains(case)):
        if d["p"].par:
            continue
        e = _Exact(d, int(seed) * 64 + k, at_rest)
        for _ in range(case["steps"]):
            e.step()
        rho, u, phi = e.macros()[:3]
        for name, v in zip(FIELDS, (rho, u[0], u[1], u[2], phi)):
            got[name].append(v.reshape(-1).cpu())
    return dict(free={k: torch.cat(v) for k, v in got.items()}, held=None, motion=None)
