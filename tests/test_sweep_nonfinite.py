"""Not-a-number and coincident inputs of the window sweep: what is not finite
in the oracle's rates is not finite here, and everything else agrees with
them, on the scale of the field's largest rate."""
import numpy as np
import pytest

import grasph_b200 as G
from gc_helpers import make_backend

pytestmark = pytest.mark.gpu

DX = 0.02
H = 1.3 * DX


def _build(nd, functor, kernel, spoil, wall=None):
    n = (9, 8) if nd == 2 else (6, 5, 4)
    rng = np.random.default_rng(2)
    x = np.stack([a.ravel() for a in np.meshgrid(*[(np.arange(m) + 0.5) * DX for m in n], indexing="ij")], axis=1)
    x += rng.uniform(-0.1, 0.1, x.shape) * DX
    k = {"spline": G.CubicSplineKernel, "wendland": G.WenlandC2Kernel}[kernel](H, ndims=nd)
    if functor == "fluid":
        ps = G.FluidParticleSystem("f", len(x), nd, 1000.0 * DX ** nd, 40.0)
        ps.p[:] = rng.uniform(-50.0, 500.0, ps.n)
        pfn = G.FluidPfn(0.05, 0.1, H)
    else:
        ps = G.ElastoPlasticParticleSystem("s", len(x), nd, 4 if nd == 2 else 6, 1000.0 * DX ** nd, 40.0)
        ps.stress[:] = rng.uniform(-300.0, 100.0, ps.stress.shape)
        pfn = (G.StrainRateVorticityPfn(), G.CauchyFluidPfn(0.05, 0.1, H))
    ps.x[:] = x
    ps.v[:] = rng.uniform(-1.0, 1.0, x.shape)
    ps.rho[:] = rng.uniform(990.0, 1010.0, ps.n)
    spoil(ps)
    systems, b = [ps], None
    if wall:
        # a wall with one particle where one of the system's is
        w = G.BasicParticleSystem("w", 1, nd, 1000.0 * DX ** nd, 40.0)
        w.x[:] = ps.x[7]
        w.rho[:] = 1000.0
        systems.append(w)
        b = (G.StaticBoundarySystem(w, DX) if wall == "static" else
             G.DynamicBoundarySystem(w, [0.0] * (nd - 1) + [1.0], w.x[0] - DX, 1.5))
    return G.LeapFrogTimeIntegrator(systems, [G.SystemInteraction(k, pfn, ps, b)])


def _check(build, precision, tol, fields, config=-1):
    """One sweep of every stage (a step would integrate what is not finite)."""
    runs = {}
    for name in ("oracle", "cuda"):
        lf = build()
        s = G.Session([lf], backend=make_backend(name), precision=precision if name == "cuda" else G.PRECISION_FP64)
        if name == "cuda" and config >= 0:
            s.backend.set_sweep_config(config)
        s.push()
        ps, si = lf.systems[0], lf.interactions[0]
        for q in lf.systems:
            s.sort_particles(q, 2.0 * H)
        s.create_grid(si)
        for stage in range(1, len(si.pfns) + 1):
            s.sweep(si, stage)
        s.pull()
        runs[name] = ps
    for f in fields:
        a, b = (np.asarray(getattr(runs[q], f), float) for q in ("cuda", "oracle"))
        assert np.array_equal(np.isfinite(a), np.isfinite(b)), f
        ok = np.isfinite(b)
        assert np.all(np.abs(a[ok] - b[ok]) <= tol * np.abs(b[ok]).max()), f
    return runs["oracle"]


FIELDS = {"fluid": ("dvdt", "drhodt"), "stress": ("dvdt", "drhodt", "strain_rate", "vorticity")}


@pytest.mark.parametrize("field,value", [("v", np.nan), ("rho", np.nan), ("rho", 0.0)])
@pytest.mark.parametrize("nd,functor", [(2, "fluid"), (3, "fluid"), (2, "stress"), (3, "stress")])
def test_fp64_neighbour_not_a_number(nd, functor, field, value):
    def spoil(ps):
        getattr(ps, field)[ps.n // 2] = value
    ps = _check(lambda: _build(nd, functor, "spline", spoil), G.PRECISION_FP64, 1e-12, FIELDS[functor])
    assert np.isnan(ps.dvdt).any(axis=1).sum() > 4 and np.isnan(ps.drhodt).sum() > 4


@pytest.mark.parametrize("precision", [G.PRECISION_FP64, G.PRECISION_FP32_COMPENSATED])
@pytest.mark.parametrize("kernel", ["spline", "wendland"])
@pytest.mark.parametrize("nd,functor", [(2, "fluid"), (3, "stress")])
def test_coincident(nd, functor, kernel, precision):
    def spoil(ps):
        ps.x[7] = ps.x[8]
    fields = FIELDS[functor]
    ps = _check(lambda: _build(nd, functor, kernel, spoil), precision,
                1e-12 if precision == G.PRECISION_FP64 else 1e-5, fields)
    assert np.isnan(ps.drhodt).sum() == 2


# The pair's r² is 2e-42 (a subnormal float) and 2e-312 (a subnormal double):
# its terms vanish with the distance.
@pytest.mark.parametrize("precision,sep", [(G.PRECISION_FP32_COMPENSATED, 1e-21), (G.PRECISION_FP64, 1e-156)])
@pytest.mark.parametrize("kernel", ["spline", "wendland"])
@pytest.mark.parametrize("nd,functor", [(2, "fluid"), (3, "stress")])
def test_nearly_coincident(nd, functor, kernel, precision, sep):
    def spoil(ps):
        ps.x[:] -= ps.x[8]
        ps.x[7] = 0.0
        ps.x[7, :2] = sep
    ps = _check(lambda: _build(nd, functor, kernel, spoil), precision,
                1e-12 if precision == G.PRECISION_FP64 else 1e-5, FIELDS[functor])
    assert np.isfinite(ps.dvdt).all() and np.isfinite(ps.drhodt).all()


@pytest.mark.parametrize("precision", [G.PRECISION_FP64, G.PRECISION_FP32_COMPENSATED])
@pytest.mark.parametrize("wall", ["static", "dynamic"])
@pytest.mark.parametrize("functor", ["fluid", "stress"])
def test_coincident_with_a_wall(functor, wall, precision):
    ps = _check(lambda: _build(2, functor, "spline", lambda ps: None, wall), precision,
                1e-12 if precision == G.PRECISION_FP64 else 1e-5, ("dvdt", "drhodt", *FIELDS[functor][2:]))
    assert np.isnan(ps.dvdt).any(axis=1).sum() == 1


@pytest.mark.parametrize("precision", [G.PRECISION_FP64, G.PRECISION_FP32_COMPENSATED])
def test_coincident_far_out(precision):
    """(where FP32-compensated takes FP64 differences)"""
    def spoil(ps):
        ps.x[:] += 2.0 * H * 3.0 * 2 ** 20
        ps.x[7] = ps.x[8]
    ps = _check(lambda: _build(2, "stress", "wendland", spoil), precision,
                1e-12 if precision == G.PRECISION_FP64 else 1e-5, FIELDS["stress"])
    assert np.isnan(ps.drhodt).sum() == 2


@pytest.mark.parametrize("config", range(4))
@pytest.mark.parametrize("kernel", ["spline", "wendland"])
@pytest.mark.parametrize("nd,functor", [(2, "fluid"), (3, "stress")])
def test_an_ulp_apart(nd, functor, kernel, config):
    """Positions that differ, but by less than an FP32 pair holds: no NaN."""
    def spoil(ps):
        ps.x[7] = ps.x[8]
        ps.x[7, 0] = np.nextafter(ps.x[8, 0], 1.0)
    ps = _check(lambda: _build(nd, functor, kernel, spoil), G.PRECISION_FP32_COMPENSATED, 1e-5, FIELDS[functor],
                config)
    assert np.isfinite(ps.dvdt).all() and np.isfinite(ps.drhodt).all()
