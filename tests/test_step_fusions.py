"""The half step taken with the sort's gather and the boxes left by the full
step: several instances stepped together, their boxes kept from step to step,
give the bits of each instance alone, one step a call, with its state pulled
and pushed in between (which drops the kept boxes).  Sizes around one warp,
one block and several tiles a block; updaters that overwrite some fields in
every instance and others in one only."""
import numpy as np
import pytest

import grasph_b200 as G
from gc_helpers import make_backend

pytestmark = pytest.mark.gpu


def _water(n, seed, k):
    rng = np.random.default_rng(seed)
    dx = n ** (-1.0 / 3.0)
    ps = G.FluidParticleSystem("w", n, 3, 1000.0 * dx**3, 20.0, source_v=[0.0, 0.0, -9.81],
                               state_updater=(G.TaitEOSUpdater(1000.0, 20.0) if k != "linear"
                                              else G.LinearEOSUpdater(1000.0),))
    h = 1.5 * dx
    pfn = G.FluidPfn(0.1, 0.1, h)
    return _start(ps, rng, G.SystemInteraction(G.CubicSplineKernel(h, ndims=3), pfn, ps))


def _soil(n, seed, k):
    rng = np.random.default_rng(seed)
    dx = n**-0.5
    fields = ("strain_rate", "vorticity") if k else ("strain_rate",)
    ps = G.ElastoPlasticParticleSystem("s", n, 2, 4, 1000.0 * dx * dx, 20.0, source_v=[0.0, -9.81],
                                       state_updater=(G.ZeroFieldUpdater(*fields), None))
    h = 1.5 * dx
    pfns = (G.StrainRateVorticityPfn(), G.CauchyFluidPfn(0.1, 0.1, h))
    return _start(ps, rng, G.SystemInteraction(G.CubicSplineKernel(h, ndims=2), pfns, ps))


def _start(ps, rng, inter):
    ps.x[:] = rng.uniform(0.0, 1.0, ps.x.shape)
    ps.v[:] = 0.1 * rng.standard_normal(ps.v.shape)
    ps.rho[:] = 1000.0 + rng.standard_normal(ps.n)
    if hasattr(ps, "vorticity"):
        ps.vorticity[:] = rng.standard_normal(ps.vorticity.shape)
        ps.stress[:] = rng.standard_normal(ps.stress.shape)
    return G.LeapFrogTimeIntegrator([ps], [inter])


@pytest.mark.parametrize("build,sizes,kinds", [
    (_water, (1, 31, 257, 4000), ("tait",) * 4),
    (_water, (260, 33), ("linear",) * 2),
    (_water, (160000,), ("tait",)),
    (_soil, (256, 1, 700), (1, 1, 1)),
    (_soil, (300, 40, 255), (1, 0, 1)),
])
def test_steps_together_are_the_steps_alone(build, sizes, kinds):
    steps, cfl = 6, 0.05
    make = lambda: [build(n, n, k) for n, k in zip(sizes, kinds)]  # noqa: E731
    together, alone = make(), make()
    s = G.Session(together, backend=make_backend("cuda"))
    s.push()
    s.step(steps, cfl)
    s.pull()
    for lf, ref in zip(together, alone):
        t = G.Session([ref], backend=make_backend("cuda"))
        for _ in range(steps):
            t.push()
            t.step(1, cfl)
            t.pull()
        for name, _ in ref.systems[0].particle_fields():
            a, b = getattr(lf.systems[0], name), getattr(ref.systems[0], name)
            assert np.isfinite(a).all(), name
            assert np.array_equal(a, b), name
