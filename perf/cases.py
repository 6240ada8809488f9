"""Performance cases of the framework: the work a simulation program gives it.

A case is one stretch of a running simulation: `steps` leapfrog steps of a
Session whose state is on the device, then the moving systems' fields read
back to the host, as a program does between two saves.  The families are the
repository's own benchmark configurations: dam breaks in a tank (2-D and 3-D,
dynamic or Lennard-Jones walls), Drucker-Prager column collapses with a
ghost-mirrored wall, many columns packed into one Session, and a Server
working through a mix of requests.  Plain FP64 runs hold Float64 systems; the
FP32-compensated ones hold Float32 systems (their results are of that
accuracy).  The particles start disordered (jittered off the lattice, with a
swirling velocity), as they are in the middle of a run.
"""
import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "grasph.jl_b200"))

import grasph_b200 as G  # noqa: E402

GRAVITY = 9.81
# short time steps: thousands of steps in a row stay in the first part of the
# collapse, before the water has crossed the tank and splashes
WATER_CFL = 0.01
WATER_FIELDS = ("x", "v", "rho", "dvdt", "drhodt", "p", "id")
SOIL_FIELDS = ("x", "v", "rho", "dvdt", "drhodt", "stress", "strain_rate", "vorticity", "strain", "strain_p", "id")
# accepted unordered pairs per particle inside the lattice, and FLOPs of one
# pair as the reference evaluates it (bench.py's count for the fluid functor;
# strain rate, vorticity and Cauchy terms together for the soil)
PAIRS = {("water", 2): 9.0, ("water", 3): 29.0, ("soil", 2): 14.0}
PAIR_FLOPS = {("water", 2): 70.0, ("water", 3): 86.0, ("soil", 2): 130.0}


def listed():
    return [
        # the smoke test's dam break: nothing but launches and their latency
        dict(name="water2d_288_fp64", kind="water", nx=12, ny=24, nz=0, dx=0.05, wall="dynamic", precision="fp64",
             steps=100),
        # the 2-D dam break configuration, in both precisions
        dict(name="water2d_5000_fp64", kind="water", nx=50, ny=100, nz=0, dx=0.02, wall="dynamic", precision="fp64",
             steps=100),
        dict(name="water2d_5000_fp32c", kind="water", nx=50, ny=100, nz=0, dx=0.02, wall="dynamic",
             precision="fp32c", steps=100),
        # an ordinary 3-D run of odd sizes in a Lennard-Jones box (the dambreak_3d.jl layout)
        dict(name="water3d_lj_18k_fp32c", kind="water", nx=31, ny=13, nz=45, dx=0.5, wall="static",
             precision="fp32c", steps=100),
        # a mid-sized 3-D dam break in plain FP64
        dict(name="water3d_224k_fp64", kind="water", nx=60, ny=37, nz=101, dx=0.0163, wall="dynamic",
             precision="fp64", steps=50),
        # the 3-D dam break configuration: a million fluid particles
        dict(name="water3d_1m_fp32c", kind="water", nx=100, ny=50, nz=200, dx=0.01, wall="dynamic",
             precision="fp32c", steps=150),
        # a small column of odd sizes (the low end of the batched configuration)
        dict(name="soil_2013_fp32c", kind="soil", nx=61, ny=33, dx=0.002, precision="fp32c", steps=100),
        # the column collapse configuration, in both precisions
        dict(name="soil_80k_fp32c", kind="soil", nx=400, ny=200, dx=0.0005, precision="fp32c", steps=100),
        dict(name="soil_80k_fp64", kind="soil", nx=400, ny=200, dx=0.0005, precision="fp64", steps=50),
        # a quarter of the batched configuration: 64 columns of 2,000 to 60,000 particles in one Session
        dict(name="soils_64_fp32c", kind="soils", count=64, nmin=2000, nmax=60000, dx=0.0005, mix=20261203,
             precision="fp32c", steps=75),
        # a server working through ten requests of both kinds, from submission to results
        dict(name="serve_10_fp32c", kind="serve", soils=7, waters=3, nmin=5000, nmax=60000, dx=0.0005, mix=11,
             precision="fp32c", steps=100),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same families: sizes spread over their logarithm."""
    kind = rng.choice(["water2", "water3", "water3", "lj", "soil", "soil", "soils"])
    precision = rng.choice(["fp32c", "fp32c", "fp64"])
    if kind == "water2":
        n = _log_int(rng, 250, 120_000)
        nx = max(5, round(math.sqrt(n / rng.uniform(0.7, 3.0))))
        return dict(kind="water", nx=nx, ny=max(5, n // nx), nz=0, dx=1.0 / nx, wall="dynamic", precision=precision,
                    steps=rng.choice([50, 100]))
    if kind in ("water3", "lj"):
        n = _log_int(rng, 2_000, (700_000 if kind == "water3" else 60_000) // (4 if precision == "fp64" else 1))
        side = n ** (1.0 / 3.0)
        nx = max(5, round(side * rng.uniform(0.7, 1.3)))
        ny = max(5, round(side * rng.uniform(0.4, 1.0)))
        lj = kind == "lj"
        return dict(kind="water", nx=nx, ny=ny, nz=max(5, n // (nx * ny)), dx=0.5 if lj else 1.0 / nx,
                    wall="static" if lj else "dynamic", precision=precision, steps=rng.choice([25, 50]))
    if kind == "soil":
        n = _log_int(rng, 1_000, 200_000)
        nx = max(8, round(math.sqrt(n * rng.uniform(0.25, 2.0))))
        return dict(kind="soil", nx=nx, ny=max(8, n // nx), dx=0.0005, precision=precision,
                    steps=rng.choice([50, 100]))
    return dict(kind="soils", count=rng.randint(3, 40), nmin=1000, nmax=_log_int(rng, 4000, 40000), dx=0.0005,
                mix=rng.randrange(1 << 20), precision=precision, steps=25)


# ------------------------------------------------------------------ model

def _real(case):
    return np.float32 if case["precision"] == "fp32c" else np.float64


def _jitter(x, dx, rng, amount=0.1):
    return x + rng.uniform(-amount, amount, x.shape) * dx


def _swirl(x, rng, speed):
    """A smooth swirling velocity with a little noise."""
    nd = x.shape[1]
    k = 2.0 * math.pi / max(float(np.ptp(x[:, 0])), 1e-12)
    ph = rng.uniform(0.0, 2.0 * math.pi, nd)
    v = np.stack([np.sin(k * x[:, (d + 1) % nd] + ph[d]) for d in range(nd)], axis=1)
    return speed * (v + 0.1 * rng.standard_normal(x.shape))


def _grid(*axes):
    return np.stack([a.ravel() for a in np.meshgrid(*axes, indexing="ij")], axis=1)


def _wall_faces(box, dx, layers, reach):
    """Wall particles of the box [0, box] face by face, `layers` deep: (points, inward normal, plane point)."""
    nd = len(box)
    n = [int(round(b / dx)) for b in box]
    inner = [(np.arange(m) + 0.5) * dx for m in n]
    wide = [(np.arange(-reach, m + reach) + 0.5) * dx for m in n]
    out = []
    for axis in range(nd - 1, -1, -1):  # each pair spans the thickness of those after it
        spans = [wide[d] if d < axis else inner[d] for d in range(nd)]
        for high in (False, True):
            lay = (np.arange(layers) + 0.5) * dx
            pos = box[axis] + lay if high else -lay
            pts = _grid(*[pos if d == axis else spans[d] for d in range(nd)])
            normal, point = np.zeros(nd), np.zeros(nd)
            normal[axis] = -1.0 if high else 1.0
            point[axis] = box[axis] if high else 0.0
            out.append((pts, normal, point))
    return out


def _water(case, rng):
    """A dam break: a block of fluid in a corner of a tank four blocks long."""
    T = _real(case)
    nd = 3 if case["nz"] else 2
    n = [case["nx"], case["ny"], case["nz"]][:nd]
    dx, static = case["dx"], case["wall"] == "static"
    box = [4 * n[0] * dx] + [2 * m * dx for m in n[1:]]
    height = n[-1] * dx
    c = 10.0 * math.sqrt(2.0 * GRAVITY * height)
    h, rho0, gamma = T(1.2 * dx), 1000.0, 7.0
    mass = T(rho0 * dx ** nd)
    x = _jitter(_grid(*[(np.arange(m) + 0.5) * dx for m in n]), dx, rng, 0.05 if static else 0.1)
    source = np.zeros(nd)
    source[-1] = -GRAVITY
    fluid = G.FluidParticleSystem("fluid", len(x), nd, mass, T(c), dtype=T, source_v=source,
                                  state_updater=G.TaitEOSUpdater(T(rho0), gamma=T(gamma)))
    fluid.x[:] = x
    fluid.v[:] = _swirl(x, rng, 0.02 * c)
    fluid.rho[:] = rho0 * (1.0 + gamma * GRAVITY * (height - x[:, -1]) / c ** 2) ** (1.0 / gamma)
    kernel = G.CubicSplineKernel(h, ndims=nd)
    pfn = G.FluidPfn(T(0.01), T(0.0), h)
    systems, inters = [fluid], [G.SystemInteraction(kernel, pfn, fluid)]
    faces = _wall_faces(box, dx, 1 if static else 3, 1 if static else 3)
    if static:
        faces = [(np.concatenate([f[0] for f in faces]), None, None)]
    for pts, normal, point in faces:
        ps = G.BasicParticleSystem("wall", len(pts), nd, mass, T(c), dtype=T)
        ps.x[:] = pts
        ps.rho[:] = rho0
        systems.append(ps)
        wall = G.StaticBoundarySystem(ps, dx) if static else G.DynamicBoundarySystem(ps, normal, point, 3.0)
        inters.append(G.SystemInteraction(kernel, pfn, fluid, wall))
    return G.LeapFrogTimeIntegrator(systems, inters), WATER_CFL


def _soil(case, rng, nx, ny, phi_deg=19.8, young=0.84e6):
    """A granular column on a dynamic floor against a ghost-mirrored wall."""
    T = _real(case)
    dx, rho0, nu, phi = case["dx"], 2650.0, 0.3, math.radians(phi_deg)
    c = math.sqrt(young * (1 - nu) / (rho0 * (1 + nu) * (1 - 2 * nu)))
    h, mass = T(1.5 * dx), T(rho0 * dx * dx)
    x = _jitter(_grid((np.arange(nx) + 0.5) * dx, (np.arange(ny) + 0.5) * dx), dx, rng)
    soil = G.ElastoPlasticParticleSystem(
        "soil", len(x), 2, 4, mass, T(c), dtype=T, source_v=[0.0, -GRAVITY],
        state_updater=(G.ZeroFieldUpdater("strain_rate", "vorticity"),
                       G.ElastoPlasticStressUpdater(T(young), T(nu), T(phi), T(0.0), T(0.0))))
    soil.x[:] = x
    soil.v[:] = _swirl(x, rng, 0.005 * c)
    soil.rho[:] = rho0
    syy = -rho0 * GRAVITY * (ny * dx - np.minimum(x[:, 1], ny * dx))
    k0 = 1.0 - math.sin(phi)
    soil.stress[:] = np.stack([k0 * syy, syy, k0 * syy, 0.0 * syy], axis=1)
    nb = int(round(max(2.5 * nx, nx + 20)))
    floor = G.BasicParticleSystem("floor", 3 * (nb + 3), 2, mass, T(c), dtype=T)
    floor.x[:] = _grid((np.arange(nb + 3) - 2.5) * dx, -(np.arange(3) + 0.5) * dx)
    floor.rho[:] = rho0
    ghost = G.GhostParticleSystem(soil, G.GhostCopier("stress"))
    entry = G.GhostEntry(ghost, 3.0 * float(h), ((1.0, 0.0), (0.0, 0.0)), capacity=soil.n)
    kernel = G.CubicSplineKernel(h, ndims=2)
    pfns = (G.StrainRateVorticityPfn(), G.CauchyFluidPfn(T(0.1), T(0.1), h))
    inters = [G.SystemInteraction(kernel, pfns, soil),
              G.SystemInteraction(kernel, pfns, soil, G.DynamicBoundarySystem(floor, (0.0, 1.0), (0.0, 0.0), 3.0)),
              G.SystemInteraction(kernel, pfns, soil, ghost)]
    return G.LeapFrogTimeIntegrator([soil, floor], inters, ghosts=(entry,)), 0.1


def _soil_shapes(case, count):
    """Sizes, friction angles and stiffnesses of a mix of columns (the case's own draw)."""
    mix = np.random.default_rng(case["mix"])
    out = []
    for _ in range(count):
        n = math.exp(mix.uniform(math.log(case["nmin"]), math.log(case["nmax"])))
        nx = max(8, int(round(math.sqrt(n / mix.uniform(0.5, 4.0)))))
        out.append((nx, max(8, int(round(n / nx))), mix.uniform(25.0, 40.0), mix.uniform(0.5e6, 5.0e6)))
    return out


def _water_shapes(case, count):
    mix = np.random.default_rng(case["mix"] + 1)
    out = []
    for _ in range(count):
        n = math.exp(mix.uniform(math.log(case["nmin"]), math.log(case["nmax"])))
        k = max(4, int(round((n / 4.0) ** (1.0 / 3.0))))
        out.append(dict(nx=2 * k, ny=k, nz=max(5, int(round(n / (2 * k * k)))), dx=1.0 / (2 * k), wall="dynamic",
                        precision=case["precision"]))
    return out


def _models(case, seed):
    """The case's simulations: soils and waters, each a list of (integrator, CFL)."""
    rng = np.random.default_rng([seed, 7])
    if case["kind"] == "water":
        return [], [_water(case, rng)]
    if case["kind"] == "soil":
        return [_soil(case, rng, case["nx"], case["ny"])], []
    count = case["count"] if case["kind"] == "soils" else case["soils"]
    waters = _water_shapes(case, case["waters"]) if case["kind"] == "serve" else []
    return [_soil(case, rng, *s) for s in _soil_shapes(case, count)], [_water(w, rng) for w in waters]


def _packed(models, fields):
    """The moving systems' fields as slices of one array per field."""
    systems = [lf.systems[0] for lf, _ in models]
    out = {}
    for name in fields if models else ():
        out[name] = np.concatenate([getattr(ps, name) for ps in systems])
        at = 0
        for ps in systems:
            setattr(ps, name, out[name][at:at + ps.n])
            at += ps.n
    return out


def prepare(case, seed):
    soils, waters = _models(case, seed)
    state = dict(case=case, models=soils + waters, out=dict(soil=_packed(soils, SOIL_FIELDS),
                                                             water=_packed(waters, WATER_FIELDS)))
    precision = G.PRECISION_FP32_COMPENSATED if case["precision"] == "fp32c" else G.PRECISION_FP64
    if case["kind"] == "serve":
        state["server"] = G.Server(precision=precision)
    else:
        state["session"] = G.Session([lf for lf, _ in state["models"]], precision=precision)
        state["session"].push()
    return state


def run(state):
    steps, models = state["case"]["steps"], state["models"]
    if "server" in state:
        server = state["server"]
        requests = [server.submit(lf, steps, cfl) for lf, cfl in models]
        done = (G.Server.DONE, G.Server.FAILED)
        while not all(server.poll(req)["state"] in done for req in requests):
            server.pump()
        for req in requests:
            server.fetch(req)
            server.release(req)
    else:
        session = state["session"]
        session.step(steps, models[0][1])
        session.pull(with_ghosts=False, systems=[lf.systems[0] for lf, _ in models])
    return state["out"]


def _sizes(case):
    """(family, particles, dimensions) of each simulation of the case."""
    if case["kind"] == "water":
        nd = 3 if case["nz"] else 2
        return [("water", case["nx"] * case["ny"] * max(1, case["nz"]), nd)]
    if case["kind"] == "soil":
        return [("soil", case["nx"] * case["ny"], 2)]
    count = case["count"] if case["kind"] == "soils" else case["soils"]
    out = [("soil", nx * ny, 2) for nx, ny, _, _ in _soil_shapes(case, count)]
    if case["kind"] == "serve":
        out += [("water", w["nx"] * w["ny"] * w["nz"], 3) for w in _water_shapes(case, case["waters"])]
    return out


def work(case):
    """Per step every moving particle's state read once and written once (x,
    v, rho and their rates, p; the soil's stress and strains too), and the
    pair terms of every unordered pair."""
    total_bytes = flops = 0.0
    for family, n, nd in _sizes(case):
        doubles = 3 * nd + 3 if family == "water" else 3 * nd + 2 + 4 * 4 + 1
        total_bytes += 2.0 * 8.0 * doubles * n * case["steps"]
        flops += n * PAIRS[family, nd] * PAIR_FLOPS[family, nd] * case["steps"]
    return {"bytes": total_bytes, "flops": flops}


# --------------------------------------------------- the same in 64 bits

def _t(a):
    return torch.as_tensor(np.asarray(a, dtype=np.float64), device="cuda" if torch.cuda.is_available() else "cpu")


def _strips(ax, ak, bx, bk, h, same):
    """Every pair (i of a, j of b, xi - xj, r²) of one instance closer than 2h, in parts."""
    nd = ax.shape[1]
    ca = torch.floor(ax / (2.0 * h[ak])[:, None]).long()
    cb = torch.floor(bx / (2.0 * h[bk])[:, None]).long()
    lo = torch.minimum(ca.min(0).values, cb.min(0).values) - 1
    ext = torch.maximum(ca.max(0).values, cb.max(0).values) - lo + 2

    def flat(c, k):
        f = k
        for d in range(nd):
            f = f * ext[d] + (c[:, d] - lo[d])
        return f

    kb, order = torch.sort(flat(cb, bk), stable=True)
    cells = int(h.numel() * torch.prod(ext).item())
    start = torch.zeros(cells + 4, dtype=torch.long, device=ax.device)
    start[1:cells + 1] = torch.cumsum(torch.bincount(kb, minlength=cells), 0)
    start[cells + 1:] = start[cells]
    offsets = [(o,) for o in (-1, 0, 1)] if nd == 2 else [(o, q) for o in (-1, 0, 1) for q in (-1, 0, 1)]
    for off in offsets:
        key = flat(ca + torch.tensor(off + (-1,), device=ax.device), ak)
        first, n = start[key], start[key + 3] - start[key]
        i = torch.repeat_interleave(torch.arange(len(ax), device=ax.device), n)
        j = order[first[i] + torch.arange(len(i), device=ax.device) - (torch.cumsum(n, 0) - n)[i]]
        d = ax[i] - bx[j]
        rr = (d * d).sum(1)
        keep = rr < (4.0 * h * h)[ak][i]
        if same:
            keep &= i != j
        i, j, d, rr = i[keep], j[keep], d[keep], rr[keep]
        if len(i):
            yield i, j, d, rr


def _gradient(d, rr, h, nd):
    """The cubic spline's gradient at pairs of one instance's h each."""
    r = torch.sqrt(rr)
    q = r / h
    norm = 10.0 / (7.0 * math.pi * h * h) if nd == 2 else 1.0 / (math.pi * h ** 3)
    dw = norm * -3.0 * (0.25 * torch.clamp(2.0 - q, min=0.0) ** 2 - torch.clamp(1.0 - q, min=0.0) ** 2)
    return (dw / (r * h))[:, None] * d


def _viscosity(d, dv, rr, h, ri, rj, c, alpha, beta):
    vr = torch.clamp((d * dv).sum(1), max=0.0)
    mu = h * vr / (rr + 0.01 * h * h)
    return (beta * mu - alpha * c) * mu / (0.5 * ri * rj)


def _stress_force(s, g, over):
    return torch.stack([s[:, 0] * g[:, 0] + s[:, 3] * g[:, 1], s[:, 3] * g[:, 0] + s[:, 1] * g[:, 1]], 1) * over


def _mirrored(x, v, bx, normal, point, i, j):
    """A dynamic wall particle's velocity as its neighbour i sees it."""
    da, db = (x[i] - point) @ normal, (bx[j] - point) @ normal
    return -torch.clamp(torch.abs(db / da), max=3.0)[:, None] * v[i]


class _Sim:
    """Simulations of one family side by side, in 64 bits: `k` is each particle's instance."""

    def __init__(self, models):
        systems = [lf.systems[0] for lf, _ in models]
        self.n = [ps.n for ps in systems]
        self.k = torch.repeat_interleave(torch.arange(len(models)), torch.tensor(self.n)).to(_t(0.0).device)
        self.h = _t([float(lf.interactions[0].kernel.h) for lf, _ in models])
        self.c = _t([float(ps.c) for ps in systems])
        self.mass = _t([float(ps.mass) for ps in systems])
        self.dt = _t([cfl for _, cfl in models]) * self.h / self.c
        self.source = _t(systems[0].source_v)
        for name in ("x", "v", "rho", "dvdt", "drhodt"):
            setattr(self, name, torch.cat([_t(getattr(ps, name)) for ps in systems]))
        self.nd = self.x.shape[1]
        self.carried = ["x", "v", "rho", "dvdt", "drhodt", "k"]
        walls = list(zip(*[[it.system_b for it in lf.interactions if isinstance(
            it.system_b, (G.DynamicBoundarySystem, G.StaticBoundarySystem))] for lf, _ in models]))
        self.walls = [(torch.cat([_t(w.inner.x) for w in ws]),
                       torch.repeat_interleave(torch.arange(len(ws)), torch.tensor([w.inner.n for w in ws])).to(
                           self.k.device), ws[0]) for ws in walls]

    def sort(self):
        """Stable order by cell, the first dimension outermost."""
        key = torch.floor(self.x / (2.0 * self.h[self.k])[:, None]).long()
        key -= key.min(0).values
        ext = key.max(0).values + 1
        flat = self.k
        for d in range(self.nd):
            flat = flat * ext[d] + key[:, d]
        order = torch.sort(flat, stable=True).indices
        for name in self.carried:
            setattr(self, name, getattr(self, name)[order])

    def step(self):
        self.sort()
        dt = self.dt[self.k]
        v0, rho0 = self.v, self.rho
        self.v = self.v + 0.5 * dt[:, None] * self.dvdt
        self.rho = self.rho + 0.5 * dt * self.drhodt
        self.dvdt = self.source.expand_as(self.v).clone()
        self.drhodt = torch.zeros_like(self.rho)
        self.rates(dt)
        self.v = v0 + dt[:, None] * self.dvdt
        self.rho = rho0 + dt * self.drhodt
        self.x = self.x + dt[:, None] * self.v

    def outputs(self, fields):
        return {name: None if name == "id" else getattr(self, name).cpu().numpy() for name in fields}


class _Water(_Sim):
    def __init__(self, models):
        super().__init__(models)
        pfn = models[0][0].interactions[0].pfns[0]
        self.alpha, self.beta = float(pfn.art_visc_alpha), float(pfn.art_visc_beta)
        self.p = torch.zeros_like(self.rho)

    def rates(self, dt):
        k, x, v, rho = self.k, self.x, self.v, self.rho
        self.p = (1000.0 * self.c * self.c / 7.0)[k] * ((rho / 1000.0) ** 7 - 1.0)
        pr = self.p / (rho * rho)
        for i, j, d, rr in _strips(x, k, x, k, self.h, True):
            h, c, m = self.h[k[i]], self.c[k[i]], self.mass[k[i]]
            g, dv = _gradient(d, rr, h, self.nd), v[i] - v[j]
            s = m * (-(pr[i] + pr[j]) - _viscosity(d, dv, rr, h, rho[i], rho[j], c, self.alpha, self.beta))
            self.dvdt.index_add_(0, i, s[:, None] * g)
            self.drhodt.index_add_(0, i, m * (dv * g).sum(1))
        for bx, bk, wall in self.walls:
            static = isinstance(wall, G.StaticBoundarySystem)
            for i, j, d, rr in _strips(x, k, bx, bk, self.h, False):
                h, c, m = self.h[k[i]], self.c[k[i]], self.mass[k[i]]
                g = _gradient(d, rr, h, self.nd)
                if static:
                    visc = _viscosity(d, v[i], rr, h, rho[i], 1000.0, c, self.alpha, self.beta)
                    ratio = wall.lj_cutoff / torch.sqrt(rr)
                    lj = torch.where(ratio > 1.0, 0.01 * c * c * (ratio ** 12 - ratio ** 6) / rr, 0.0)
                    self.dvdt.index_add_(0, i, (-m * visc)[:, None] * g + lj[:, None] * d)
                    continue
                dv = v[i] - _mirrored(x, v, bx, _t(wall.boundary_normal), _t(wall.boundary_point), i, j)
                visc = _viscosity(d, dv, rr, h, rho[i], rho[i], c, self.alpha, self.beta)
                self.dvdt.index_add_(0, i, (m * (-2.0 * pr[i] - visc))[:, None] * g)
                self.drhodt.index_add_(0, i, m * (dv * g).sum(1))


class _Soil(_Sim):
    def __init__(self, models):
        super().__init__(models)
        systems = [lf.systems[0] for lf, _ in models]
        for name in ("stress", "strain_rate", "vorticity", "strain", "strain_p"):
            setattr(self, name, torch.cat([_t(getattr(ps, name)) for ps in systems]))
            self.carried.append(name)
        pfn = models[0][0].interactions[0].pfns[1]
        self.alpha, self.beta = float(pfn.art_visc_alpha), float(pfn.art_visc_beta)
        ups = [ps.state_updater[1] for ps in systems]
        self.young, self.nu = _t([float(u.E) for u in ups]), float(ups[0].nu)
        sphi = torch.sin(_t([float(u.phi) for u in ups]))
        self.a_phi = 2.0 * sphi / (math.sqrt(3.0) * (3.0 - sphi))

    def rates(self, dt):
        k, x, v, rho = self.k, self.x, self.v, self.rho
        src = torch.nonzero((x[:, 0] > 0.0) & (x[:, 0] <= 3.0 * self.h[k])).ravel()
        flip = torch.tensor([-1.0, 1.0], dtype=torch.float64, device=x.device)
        gx, gv, gk, grho, gstress = x[src] * flip, v[src] * flip, k[src], rho[src], self.stress[src]
        normal, point = _t([0.0, 1.0]), _t([0.0, 0.0])
        floor, fk, _ = self.walls[0]

        def pairs():
            for i, j, d, rr in _strips(x, k, x, k, self.h, True):
                yield "self", i, j, d, rr
            for i, j, d, rr in _strips(x, k, floor, fk, self.h, False):
                yield "floor", i, j, d, rr
            for i, j, d, rr in _strips(x, k, gx, gk, self.h, False):
                yield "ghost", i, j, d, rr

        kept = []
        self.strain_rate = torch.zeros_like(self.strain_rate)
        self.vorticity = torch.zeros_like(self.vorticity)
        for kind, i, j, d, rr in pairs():
            g, m = _gradient(d, rr, self.h[k[i]], 2), self.mass[k[i]]
            if kind == "floor":
                vj, rj = _mirrored(x, v, floor, normal, point, i, j), rho[i]
            else:
                vj, rj = (v[j], rho[j]) if kind == "self" else (gv[j], grho[j])
            dv, f = vj - v[i], m / rj
            sr = torch.stack([dv[:, 0] * g[:, 0], dv[:, 1] * g[:, 1], torch.zeros_like(f),
                              0.5 * (dv[:, 0] * g[:, 1] + dv[:, 1] * g[:, 0])], 1)
            self.strain_rate.index_add_(0, i, sr * f[:, None])
            self.vorticity.index_add_(0, i, 0.5 * (dv[:, 0] * g[:, 1] - dv[:, 1] * g[:, 0]) * f)
            kept.append((kind, i, j, d, rr, g, dv, rj))
        self.yield_stress(dt)
        for kind, i, j, d, rr, g, dv, rj in kept:
            h, c, m = self.h[k[i]], self.c[k[i]], self.mass[k[i]]
            sj = {"self": lambda: self.stress[j], "floor": lambda: self.stress[i], "ghost": lambda: gstress[j]}[kind]()
            visc = _viscosity(d, -dv, rr, h, rho[i], rj, c, self.alpha, self.beta)
            force = _stress_force(self.stress[i], g, (1.0 / rho[i] ** 2)[:, None]) + _stress_force(
                sj, g, (1.0 / rj ** 2)[:, None]) - visc[:, None] * g
            self.dvdt.index_add_(0, i, m[:, None] * force)
            self.drhodt.index_add_(0, i, m * (-dv * g).sum(1))

    def yield_stress(self, dt):
        """Drucker-Prager with zero dilatancy and cohesion, plane strain."""
        k, s, nu = self.k, self.stress, self.nu
        d0, a_phi = (self.young / ((1 + nu) * (1 - 2 * nu)))[k], self.a_phi[k]
        w = self.vorticity * dt

        def elastic(e):
            tr = nu * (e[:, 0] + e[:, 1] + e[:, 2])
            lin = (1 - 2 * nu) * e
            return d0[:, None] * (lin + torch.stack([tr, tr, tr, torch.zeros_like(tr)], 1))

        de = self.strain_rate * dt[:, None]
        spin = torch.stack([-2 * s[:, 3] * w, 2 * s[:, 3] * w, torch.zeros_like(w), (s[:, 0] - s[:, 1]) * w], 1)
        ds = elastic(de) + spin
        trial = s + ds
        i1 = trial[:, :3].sum(1)
        dev = trial - torch.stack([i1 / 3, i1 / 3, i1 / 3, torch.zeros_like(i1)], 1)
        weight = torch.tensor([1.0, 1.0, 1.0, 2.0], dtype=torch.float64, device=s.device)
        j2 = torch.sqrt(0.5 * (weight * dev * dev).sum(1))
        f = a_phi * i1 + j2
        plastic = f > 0.0
        flow = dev / torch.where(plastic, 2.0 * j2, torch.ones_like(j2))[:, None]
        df = flow + a_phi[:, None] * torch.tensor([1.0, 1.0, 1.0, 0.0], dtype=torch.float64, device=s.device)
        lam = f / (weight * df * elastic(flow)).sum(1)
        dep = torch.where(plastic[:, None], lam[:, None] * flow, torch.zeros_like(flow))
        out = trial - torch.where(plastic[:, None], elastic(dep), torch.zeros_like(dep))
        self.stress = torch.where((out[:, :3].sum(1) > 0.0)[:, None], torch.zeros_like(out), out)
        self.strain = self.strain + de
        self.strain_p = self.strain_p + dep


def exact(case, seed):
    soils, waters = _models(case, seed)
    out = {"soil": {}, "water": {}}
    for name, models, sim, fields in (("soil", soils, _Soil, SOIL_FIELDS), ("water", waters, _Water, WATER_FIELDS)):
        # simulations of one shape of model advance together
        if not models:
            continue
        s = sim(models)
        for _ in range(case["steps"]):
            s.step()
        out[name] = s.outputs(fields)
    return out
