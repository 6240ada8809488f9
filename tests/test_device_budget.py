"""Steps that outgrow the device budget: every budget between what the first
step takes and what a step of a spread-out state would, so that each of its
allocations is the one that fails."""
import numpy as np
import pytest

import grasph_b200 as G

pytestmark = pytest.mark.gpu

DX = 0.02


def _build(kind):
    rng = np.random.default_rng(4)
    i, j = np.meshgrid(np.arange(20), np.arange(12), indexing="ij")
    x = np.stack([i.ravel(), j.ravel()], axis=1) * DX + 0.011
    h = 1.3 * DX
    k = G.CubicSplineKernel(h, ndims=2)
    w = G.BasicParticleSystem("b", 40, 2, 0.4, 40.0)
    w.x[:, 0] = np.arange(40) * DX / 2
    w.x[:, 1] = -0.01
    w.rho[:] = 1000.0
    ghosts = ()
    if kind == "water":
        ps = G.FluidParticleSystem("w", len(x), 2, 0.4, 40.0, state_updater=(G.TaitEOSUpdater(1000.0, 40.0),))
        pfns = (G.FluidPfn(0.1, 0.1, h),)
        inters = []
    else:
        ps = G.ElastoPlasticParticleSystem("s", len(x), 2, 4, 0.4, 40.0)
        ps.stress[:] = rng.uniform(-300.0, 100.0, ps.stress.shape)
        pfns = (G.StrainRateVorticityPfn(), G.CauchyFluidPfn(0.1, 0.1, h))
        ghost = G.GhostParticleSystem(ps, None, G.GhostCopier("stress"))
        ghosts = (G.GhostEntry(ghost, 3.0 * h, ((1.0, 0.0), (0.0, 0.0))),)
        inters = [G.SystemInteraction(k, pfns, ps, ghost)]
    ps.x[:] = x + rng.uniform(-1e-3, 1e-3, x.shape)
    ps.v[:] = rng.uniform(-1.0, 1.0, x.shape)
    ps.rho[:] = rng.uniform(990.0, 1010.0, ps.n)
    inters += [G.SystemInteraction(k, pfns, ps),
               G.SystemInteraction(k, pfns, ps, G.DynamicBoundarySystem(w, [0.0, 1.0], [0.0, 0.0], 1.5))]
    return G.LeapFrogTimeIntegrator([ps, w], inters, ghosts=ghosts)


def _fits(call):
    """Whether a call had the memory it needs."""
    try:
        call()
    except G.GcError as e:
        assert "GC_ERR_OOM" in str(e), e
        return False
    return True


def _step(s):
    return _fits(lambda: s.step(1, 0.01))


def _tight(kind):
    """Sessions under budgets that hold the first step but not the step of
    the state just pushed."""
    budget, held = 200_000, False
    while True:
        budget += 60_000
        lf = _build(kind)
        made = []
        if not _fits(lambda: made.append(G.Session([lf], hbm_budget=budget))):
            continue
        s = made[0]
        if not _fits(s.push) or not _step(s):
            assert not held
            continue
        held = True
        s.pull()
        lf.systems[0].x[-1] += 8.0  # many more cells
        s.push()
        if _step(s):
            return
        yield lf, s
        s.backend.close()


@pytest.mark.parametrize("kind", ["water", "soil"])
def test_a_step_that_does_not_fit_fails_again(kind):
    """(on buffers that the failed one has given back)"""
    met = 0
    for lf, s in _tight(kind):
        met += 1
        assert not _step(s)
        for si in lf.interactions:
            _fits(lambda: s.create_grid(si))  # noqa: B023
            assert not _step(s)
    assert met > 5


@pytest.mark.parametrize("kind", ["water", "soil"])
def test_a_step_that_does_not_fit_leaves_the_state(kind):
    met = 0
    for lf, s in _tight(kind):
        met += 1
        before = {}
        for ps in lf.systems:
            order = np.argsort(ps.id)
            before[ps.name] = {f: np.array(getattr(ps, f))[order] for f, _ in ps.particle_fields()}
        assert not _step(s)
        s.pull()
        for ps in lf.systems:
            order = np.argsort(ps.id)
            for f, _ in ps.particle_fields():
                assert np.array_equal(getattr(ps, f)[order], before[ps.name][f]), f"{ps.name} {f}"
    assert met > 5
