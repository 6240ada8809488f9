"""The window sweep at the sizes where its chunks, masks, cutoff band and
far-away branch change: its neighbour counts are the counting sweep's in
either precision, and its rates the oracle's within rounding.

Tolerance: a pair's term takes fewer than 24 rounded FP32 operations, each
off by at most 2^-24 of the term's input magnitudes, and the compensated sum
adds no more than one; so a particle's rate is within 25·2^-24 of the sum of
its terms' magnitudes (the oracle's INPUTS shadow).  In FP64 a term takes
fewer than 40 operations on either side, and the plain sums of n terms add n:
2·(40 + n)·2^-53."""
import numpy as np
import pytest

import grasph_b200 as G
import parity
from gc_helpers import make_backend

pytestmark = pytest.mark.gpu

# points per dimension, h / spacing, jitter / spacing, offset in cells
SHAPES = {
    "one_particle": ((1, 1), 1.2, 0.0, 0),
    "one_cell": ((3, 2), 1.5, 0.1, 0),
    "columns_of_31_to_33": ((3, 97), 1.6, 0.1, 0),
    "chunks_2d": ((40, 60), 4.1, 0.1, 0),  # about 800 candidates a window
    "chunks_3d": ((14, 12, 16), 2.3, 0.1, 0),
    "on_the_cutoff_2d": ((24, 30), 1.5, 0.0, 0),
    "on_the_cutoff_3d": ((8, 7, 9), 1.5, 0.0, 0),
    "far_out": ((12, 20), 1.3, 0.1, 3 * 2 ** 20),
    "negative": ((12, 20), 1.3, 0.1, -40),
}


def _build(shape, functor, kernel):
    n, hfac, jitter, off = SHAPES[shape]
    nd, dx = len(n), 0.02
    h, c = hfac * dx, 40.0
    rng = np.random.default_rng(5)
    x = np.stack([a.ravel() for a in np.meshgrid(*[(np.arange(m) + 0.5) * dx for m in n], indexing="ij")], axis=1)
    x += rng.uniform(-jitter, jitter, x.shape) * dx + off * 2.0 * h
    k = {"spline": G.CubicSplineKernel, "wendland": G.WenlandC2Kernel}[kernel](h, ndims=nd)
    if functor == "fluid":
        ps = G.FluidParticleSystem("f", len(x), nd, 1000.0 * dx ** nd, c)
        ps.p[:] = rng.uniform(-50.0, 500.0, ps.n)
        inter = G.SystemInteraction(k, G.FluidPfn(0.05, 0.1, h, delta=0.1), ps)
    else:
        ns = 4 if nd == 2 else 6
        ps = G.ElastoPlasticParticleSystem("s", len(x), nd, ns, 1000.0 * dx ** nd, c)
        ps.stress[:] = rng.uniform(-300.0, 100.0, ps.stress.shape)
        inter = G.SystemInteraction(k, (G.StrainRateVorticityPfn(), G.CauchyFluidPfn(0.05, 0.1, h, delta=0.1)), ps)
    ps.x[:] = x
    ps.v[:] = rng.uniform(-1.0, 1.0, x.shape)
    ps.rho[:] = rng.uniform(990.0, 1010.0, ps.n)
    return G.LeapFrogTimeIntegrator([ps], [inter])


def _counts(shape, functor, kernel):
    """Every particle's neighbours, from the counting sweep."""
    lf = _build(shape, functor, kernel)
    s = G.Session([lf], backend=make_backend("cuda"))
    s.push()
    ps, si = lf.systems[0], lf.interactions[0]
    s.sort_particles(ps, 2.0 * si.kernel.h)
    s.create_grid(si)
    return s.neighbor_counts(si)


@pytest.mark.parametrize("functor", ["fluid", "stress"])
@pytest.mark.parametrize("shape", list(SHAPES))
def test_window_sweep(shape, functor):
    kernel = "wendland" if shape in ("columns_of_31_to_33", "negative") else "spline"
    runs = {}
    for name in ("oracle", "fp64", "fp32c"):
        lf = _build(shape, functor, kernel)
        prec = G.PRECISION_FP32_COMPENSATED if name == "fp32c" else G.PRECISION_FP64
        be = make_backend("oracle", track=parity.INPUTS) if name == "oracle" else make_backend("cuda")
        s = G.Session([lf], backend=be, precision=prec)
        s.push()
        s.step(1, 0.01)
        s.pull()
        runs[name] = (lf, s)
    ref, so = runs["oracle"]
    ps = ref.systems[0]
    mags = parity.oracle_magnitudes(so, ref)[id(ps)]
    scales = parity.particle_scales(ps, mags)
    counts = _counts(shape, functor, kernel)
    for name in ("fp64", "fp32c"):
        got = runs[name][0].systems[0]
        assert runs[name][1].stats()["pairs_last_step"] == counts.sum() // 2
        assert np.array_equal(ps.id, got.id)
        tol = 25 * 2.0 ** -24 if name == "fp32c" else 2.0 * (40 + counts.max()) * 2.0 ** -53
        for f in ("dvdt", "drhodt") + (("strain_rate", "vorticity") if functor == "stress" else ()):
            a, b = (np.asarray(getattr(q, f), float).reshape(ps.n, -1) for q in (got, ps))
            scale = np.max(np.asarray(scales[f]).reshape(ps.n, -1), axis=1, keepdims=True)
            worst = np.max(np.abs(a - b) / np.maximum(scale, 1e-300))
            assert np.all(np.abs(a - b) <= tol * scale), f"{name} {f}: {worst:.2e} against {tol:.2e}"
