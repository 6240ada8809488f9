"""A sweep reads the records of the state, functor and precision that it is
for: when a system's buffer grows under another system's sweep, when two
functors of one stage take turns, and when a single sweep follows a step.

Each is compared, bit by bit, with an order of the same interactions (or a
fresh session) in which every sweep finds its records where the half step or
its own pack has just put them."""
import numpy as np
import pytest

import grasph_b200 as G
from gc_helpers import make_backend

pytestmark = pytest.mark.gpu

H, DX, C0 = 0.03, 0.02, 40.0
PRECISIONS = [G.PRECISION_FP64, G.PRECISION_FP32_COMPENSATED]


def _block(ps, n, origin, seed):
    rng = np.random.default_rng(seed)
    i, j = np.meshgrid(np.arange(n[0]), np.arange(n[1]), indexing="ij")
    ps.x[:] = np.stack([i.ravel(), j.ravel()], axis=1) * DX + np.asarray(origin) + rng.uniform(-2e-3, 2e-3, ps.x.shape)
    ps.v[:] = rng.uniform(-1.0, 1.0, ps.x.shape)
    ps.rho[:] = rng.uniform(990.0, 1010.0, ps.n)
    if hasattr(ps, "stress"):
        ps.stress[:] = rng.uniform(-300.0, 100.0, ps.stress.shape)
    if hasattr(ps, "p"):
        ps.p[:] = rng.uniform(-50.0, 500.0, ps.n)
    return ps


def _soil(n, origin, seed):
    return _block(G.ElastoPlasticParticleSystem(f"s{seed}", n[0] * n[1], 2, 4, 0.4, C0), n, origin, seed)


def _water(n, origin, seed):
    return _block(G.FluidParticleSystem(f"w{seed}", n[0] * n[1], 2, 0.4, C0), n, origin, seed)


def _wall(ps, y):
    return G.DynamicBoundarySystem(ps, [0.0, 1.0], [0.0, y], 1.5)


def _session(lf, precision):
    s = G.Session([lf], backend=make_backend("cuda"), precision=precision)
    s.push()
    return s


def _equal(got, want):
    assert np.abs(got.systems[0].dvdt).max() > 0.0
    want = {ps.name: ps for ps in want.systems}
    for ps in got.systems:
        for f, _ in ps.particle_fields():
            a, b = getattr(ps, f), getattr(want[ps.name], f)
            assert np.isfinite(a).all() and np.array_equal(a, b), f"{ps.name} {f}"


def _growing(turned):
    """Soil on a moving fluid as its wall: the soil's larger records grow the
    fluid's buffer after the fluid's half step has filled it (turned: after
    the fluid's own sweep)."""
    s, w = _soil((12, 8), (0.0, 0.0), 1), _water((12, 6), (0.0, -0.12), 2)
    k = G.CubicSplineKernel(H, ndims=2)
    return G.LeapFrogTimeIntegrator([w, s] if turned else [s, w], [
        G.SystemInteraction(k, G.CauchyFluidPfn(0.1, 0.1, H), s, _wall(w, -0.01)),
        G.SystemInteraction(k, G.FluidPfn(0.1, 0.1, H), w)])


def _turns(turned):
    """One stage with strain rate, Cauchy and strain rate functors (turned:
    the Cauchy one first)."""
    s, a, b = _soil((12, 8), (0.0, 0.0), 1), _water((12, 2), (0.0, -0.04), 2), _water((12, 2), (0.0, 0.16), 3)
    k = G.CubicSplineKernel(H, ndims=2)
    inters = [G.SystemInteraction(k, G.StrainRatePfn(), s),
              G.SystemInteraction(k, G.CauchyFluidPfn(0.1, 0.1, H), s, _wall(a, -0.01)),
              G.SystemInteraction(k, G.StrainRateVorticityPfn(), s, _wall(b, 0.15))]
    if turned:
        inters = [inters[1], inters[0], inters[2]]
    return G.LeapFrogTimeIntegrator([s, a, b], inters)


@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("build", [_growing, _turns])
def test_one_step(build, precision):
    got, want = build(False), build(True)
    for lf in (got, want):
        s = _session(lf, precision)
        s.step(1, 0.01)
        s.pull()
    _equal(got, want)


@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("wall", [False, True])
def test_single_sweep_after_a_step(precision, wall):
    """The state pushed between the step and the sweep is the one swept."""
    def build(seed):
        w = _water((12, 9), (0.0, 0.0), seed)
        k = G.CubicSplineKernel(H, ndims=2)
        systems, inters = [w], [G.SystemInteraction(k, G.FluidPfn(0.1, 0.1, H), w)]
        if wall:  # a moving system that lends its positions
            systems.append(_water((12, 3), (0.0, -0.06), seed + 1))
            inters.append(G.SystemInteraction(k, G.FluidPfn(0.1, 0.1, H), w, _wall(systems[1], -0.01)))
        for i, ps in enumerate(systems):
            ps.name = f"w{i}"
        return G.LeapFrogTimeIntegrator(systems, inters)

    def sweep(lf, s):
        for ps in lf.systems:
            s.sort_particles(ps, 2.0 * H)
        for si in lf.interactions:
            s.create_grid(si)
            s.sweep(si, 1)
        s.pull()

    want = build(7)
    sweep(want, _session(want, precision))
    got, new = build(1), build(7)
    s = _session(got, precision)
    s.step(1, 0.01)
    for ps, to in zip(got.systems, new.systems):
        for f, _ in ps.particle_fields():
            getattr(ps, f)[:] = getattr(to, f)
    s.push()
    sweep(got, s)
    _equal(got, want)


@pytest.mark.parametrize("first,then", [PRECISIONS, PRECISIONS[::-1]])
def test_precision_changed_between_captured_steps(first, then):
    """(the capture of the first step in the other precision is given up when
    a record buffer has to grow, and what it had only recorded never ran)"""
    def build():
        rng = np.random.default_rng(8)
        g = np.stack([a.ravel() for a in np.meshgrid(*[np.arange(m) for m in (6, 5, 6)], indexing="ij")], axis=1)
        s = G.ElastoPlasticParticleSystem("s", len(g), 3, 6, 1000.0 * DX ** 3, C0)
        s.x[:] = g * DX + rng.uniform(-2e-3, 2e-3, g.shape) + [0.0, 0.0, DX]
        s.v[:] = rng.uniform(-1.0, 1.0, g.shape)
        s.rho[:] = rng.uniform(990.0, 1010.0, s.n)
        s.stress[:] = rng.uniform(-300.0, 100.0, s.stress.shape)
        w = G.BasicParticleSystem("w", 60, 3, 1.0, C0)
        w.x[:] = g[g[:, 2] < 2] * DX - [0.0, 0.0, DX + 1e-3]
        w.rho[:] = 1000.0
        pfns = (G.StrainRateVorticityPfn(), G.CauchyFluidPfn(0.1, 0.1, H))
        k = G.CubicSplineKernel(H, ndims=3)
        return G.LeapFrogTimeIntegrator([s, w], [
            G.SystemInteraction(k, pfns, s),
            G.SystemInteraction(k, pfns, s, G.DynamicBoundarySystem(w, [0.0, 0.0, 1.0], [0.0, 0.0, 0.0], 1.5))])

    got, want = build(), build()
    s = _session(got, first)
    s.step(24, 1e-4)  # past the tuner, into captured steps
    assert s.stats()["graph_steps"] > 0
    s.pull()
    for ps, to in zip(want.systems, got.systems):
        for f, _ in ps.particle_fields():
            getattr(ps, f)[:] = getattr(to, f)
    s.backend.set_precision(then)
    s.step(1, 1e-4)
    s.pull()
    t = _session(want, then)
    t.step(1, 1e-4)
    t.pull()
    _equal(got, want)
