"""The window sweep away from the origin: its neighbour counts and rates are
those of the same arithmetic next to it, up to where FP64 differences take
over (2^20 cells), and beyond.

Tolerance: that of the window sweep's rates (test_sweep_window.py)."""
import numpy as np
import pytest

import grasph_b200 as G
import parity
from gc_helpers import make_backend

pytestmark = pytest.mark.gpu

DX = 0.02


def _build(nd, functor, cells, wall, spread=False):
    h, c = 1.3 * DX, 40.0
    n = (16, 30) if nd == 2 else (7, 8, 10)
    rng = np.random.default_rng(3)
    x = np.stack([a.ravel() for a in np.meshgrid(*[(np.arange(m) + 0.5) * DX for m in n], indexing="ij")], axis=1)
    x += rng.uniform(-0.1, 0.1, x.shape) * DX
    # every coordinate as far out, on either side of the origin
    off = 2.0 * h * cells * np.array([1.0, -1.0, 1.0])[:nd]
    k = G.CubicSplineKernel(h, ndims=nd)
    if functor == "fluid":
        ps = G.FluidParticleSystem("f", len(x), nd, 1000.0 * DX ** nd, c)
        ps.p[:] = rng.uniform(-50.0, 500.0, ps.n)
        pfn = G.FluidPfn(0.05, 0.1, h, delta=0.1)
    else:
        ps = G.ElastoPlasticParticleSystem("s", len(x), nd, 4 if nd == 2 else 6, 1000.0 * DX ** nd, c)
        ps.stress[:] = rng.uniform(-300.0, 100.0, ps.stress.shape)
        pfn = (G.StrainRateVorticityPfn(), G.CauchyFluidPfn(0.05, 0.1, h, delta=0.1))
    ps.v[:] = rng.uniform(-1.0, 1.0, x.shape)
    ps.rho[:] = rng.uniform(990.0, 1010.0, ps.n)
    ps.x[:] = x + off
    if spread:  # every other particle as far on the other side of the middle, along x
        ps.x[:] = x
        ps.x[::2, 0] += off[0]
        ps.x[1::2, 0] -= off[0]
    systems, inters = [ps], [G.SystemInteraction(k, pfn, ps)]
    if wall:
        w = x[x[:, -1] < 3 * DX] * np.array([1.0] * (nd - 1) + [-1.0])
        b = G.BasicParticleSystem("w", len(w), nd, 1000.0 * DX ** nd, c)
        b.x[:] = w + off
        b.rho[:] = 1000.0
        systems.append(b)
        inters.append(G.SystemInteraction(k, pfn, ps,
                                          G.DynamicBoundarySystem(b, [0.0] * (nd - 1) + [1.0], off, 1.5)))
    return G.LeapFrogTimeIntegrator(systems, inters)


def _pairs(lf):
    """Accepted pairs, from the counting sweep, and the most of a particle."""
    s = G.Session([lf], backend=make_backend("cuda"))
    s.push()
    for ps in lf.systems:
        s.sort_particles(ps, 2.0 * lf.interactions[0].kernel.h)
    counts = []
    for si in lf.interactions:
        s.create_grid(si)
        counts.append(s.neighbor_counts(si))
    pairs = sum(int(c.sum()) // (1 if si.is_coupled() else 2) for c, si in zip(counts, lf.interactions))
    return pairs, max(c.max() for c in counts)


@pytest.mark.parametrize("cells", [0, 5e3, 1e4, 1e5, 9e5, 1.5e6])
@pytest.mark.parametrize("nd,functor,wall", [(2, "fluid", True), (2, "stress", False), (3, "fluid", False),
                                             (3, "stress", True)])
def test_offset(nd, functor, wall, cells):
    _check(nd, functor, cells, wall)


@pytest.mark.parametrize("cells", [1e4, 1e5, 4e5, 1.2e6])
@pytest.mark.parametrize("functor", ["fluid", "stress"])
def test_spread(functor, cells):
    """Two halves of one system, as far from the point that both count from."""
    _check(2, functor, cells, False, True)


def _check(nd, functor, *rest):
    runs = {}
    for name in ("oracle", "fp64", "fp32c"):
        lf = _build(nd, functor, *rest)
        prec = G.PRECISION_FP32_COMPENSATED if name == "fp32c" else G.PRECISION_FP64
        be = make_backend("oracle", track=parity.INPUTS) if name == "oracle" else make_backend("cuda")
        s = G.Session([lf], backend=be, precision=prec)
        s.push()
        s.step(1, 0.01)
        s.pull()
        runs[name] = (lf, s)
    ref, so = runs["oracle"]
    ps = ref.systems[0]
    scales = parity.particle_scales(ps, parity.oracle_magnitudes(so, ref)[id(ps)])
    pairs, most = _pairs(_build(nd, functor, *rest))
    for name in ("fp64", "fp32c"):
        got = runs[name][0].systems[0]
        assert runs[name][1].stats()["pairs_last_step"] == pairs
        assert np.array_equal(ps.id, got.id)
        tol = 25 * 2.0 ** -24 if name == "fp32c" else 2.0 * (40 + most) * 2.0 ** -53
        for f in ("dvdt", "drhodt") + (("strain_rate", "vorticity") if functor == "stress" else ()):
            a, b = (np.asarray(getattr(q, f), float).reshape(ps.n, -1) for q in (got, ps))
            scale = np.max(np.asarray(scales[f]).reshape(ps.n, -1), axis=1, keepdims=True)
            worst = np.max(np.abs(a - b) / np.maximum(scale, 1e-300))
            assert np.all(np.abs(a - b) <= tol * scale), f"{name} {f}: {worst:.2e} against {tol:.2e}"


@pytest.mark.parametrize("cells", [0, 7e3, 3e6])
@pytest.mark.parametrize("wall", [False, True])
def test_steps_far_out_depend_on_the_state_alone(wall, cells):
    """Captured steps in one call, and one step a call with the state pulled
    and pushed in between (FP32-compensated: the same bits)."""
    steps, cfl = 24, 0.05
    got, want = (_build(2, "fluid", cells, wall) for _ in range(2))
    s = G.Session([got], precision=G.PRECISION_FP32_COMPENSATED)
    s.push()
    s.step(steps, cfl)
    assert s.stats()["graph_steps"] > 0
    s.pull()
    t = G.Session([want], precision=G.PRECISION_FP32_COMPENSATED)
    for _ in range(steps):
        t.push()
        t.step(1, cfl)
        t.pull()
    for a, b in zip(got.systems, want.systems):
        for f, _ in a.particle_fields():
            assert np.isfinite(getattr(a, f)).all() and np.array_equal(getattr(a, f), getattr(b, f)), f"{a.name} {f}"


@pytest.mark.parametrize("cells", [0, 3e6])
def test_both_precisions_in_one_step(cells):
    """A system swept in FP64 (the S = 1 pressure form always is) that lends
    its positions to an FP32-compensated sweep in between."""
    def build():
        rng = np.random.default_rng(6)
        h = 1.3 * DX
        off = 2.0 * h * cells
        k = G.CubicSplineKernel(h, ndims=2)
        systems = []
        for name, y in (("a", 0.0), ("b", -12 * DX)):
            i, j = np.meshgrid(np.arange(14), np.arange(12), indexing="ij")
            ps = G.FluidParticleSystem(name, i.size, 2, 0.4, 40.0)
            ps.x[:] = np.stack([i.ravel(), j.ravel()], axis=1) * DX + [0.0, y] + off
            ps.x[:] += rng.uniform(-2e-3, 2e-3, ps.x.shape)
            ps.v[:] = rng.uniform(-1.0, 1.0, ps.x.shape)
            ps.rho[:] = rng.uniform(990.0, 1010.0, ps.n)
            ps.p[:] = rng.uniform(-50.0, 500.0, ps.n)
            systems.append(ps)
        a, b = systems
        wall = G.DynamicBoundarySystem(b, [0.0, 1.0], [off, off - DX / 2], 1.5)
        return G.LeapFrogTimeIntegrator(systems, [
            G.SystemInteraction(k, G.FluidPfn(0.1, 0.1, h), a),
            G.SystemInteraction(k, G.FluidPfn(0.1, 0.1, h), a, wall),
            G.SystemInteraction(k, G.FluidPfn(0.1, 0.1, h, sigma=1), b)])

    ref, lf = build(), build()
    so = G.Session([ref], backend=make_backend("oracle", track=parity.INPUTS))
    s = G.Session([lf], precision=G.PRECISION_FP32_COMPENSATED)
    for q in (so, s):
        q.push()
        q.step(1, 0.01)
        q.pull()
    pairs, most = _pairs(build())
    assert s.stats()["pairs_last_step"] == pairs
    got, ps = lf.systems[1], ref.systems[1]
    scales = parity.particle_scales(ps, parity.oracle_magnitudes(so, ref)[id(ps)])
    assert np.array_equal(got.id, ps.id)
    for f in ("dvdt", "drhodt"):
        a, b = (np.asarray(getattr(q, f), float).reshape(ps.n, -1) for q in (got, ps))
        scale = np.max(np.asarray(scales[f]).reshape(ps.n, -1), axis=1, keepdims=True)
        assert np.all(np.abs(a - b) <= 2.0 * (40 + most) * 2.0 ** -53 * scale), f


def test_instance_far_out_in_a_mix_equals_alone():
    """(FP32-compensated; a wall at rest in one instance moves in the other)"""
    def build(k):
        lf = _build(2, "fluid", 3e6 + 1e4 * k, True)
        lf.systems[1].v[:] = [0.3 * k, 0.0]
        return lf
    mix, alone = [build(k) for k in range(2)], [build(k) for k in range(2)]
    s = G.Session(mix, precision=G.PRECISION_FP32_COMPENSATED)
    s.push()
    s.step(20, 0.05)
    s.pull()
    for a, b in zip(mix, alone):
        t = G.Session([b], precision=G.PRECISION_FP32_COMPENSATED)
        t.push()
        t.step(20, 0.05)
        t.pull()
        for p, q in zip(a.systems, b.systems):
            for f, _ in p.particle_fields():
                assert np.isfinite(getattr(p, f)).all() and np.array_equal(getattr(p, f), getattr(q, f)), f"{p.name} {f}"
