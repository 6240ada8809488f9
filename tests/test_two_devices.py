"""Contexts on two devices of one process: kernel attributes belong to a
device, so the second device's sweeps need their own.  (Each device runs by
itself; nothing is shared between them.)"""
import numpy as np
import pytest
import torch

import grasph_b200 as G
from grasph_b200 import scenarios

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(torch.cuda.device_count() < 2, reason="needs two devices")]


def _soil():
    g = np.stack([a.ravel() for a in np.meshgrid(*[np.arange(6)] * 3, indexing="ij")], axis=1)
    s = G.ElastoPlasticParticleSystem("s", len(g), 3, 6, 0.008, 40.0)
    s.x[:] = g * 0.02
    s.v[:] = np.sin(3.0 * s.x)
    s.rho[:] = 1000.0
    pfns = (G.StrainRateVorticityPfn(), G.CauchyFluidPfn(0.1, 0.1, 0.026))
    return G.LeapFrogTimeIntegrator([s], [G.SystemInteraction(G.CubicSplineKernel(0.026, ndims=3), pfns, s)])


def _water():
    return scenarios.dambreak_2d(nx=12, ny=24, dx=0.05, tank=(1.5, 2.0))[0]


@pytest.mark.parametrize("build", [_soil, _water])  # over 48 KB by its records, and by an even spread of few groups
def test_same_bits_on_either_device(build):
    runs = []
    for device in (0, 1):
        lf = build()
        s = G.Session([lf], device=device)
        s.push()
        s.step(24, 1e-3)
        s.pull()
        runs.append(lf.systems[0])
    for f, _ in runs[0].particle_fields():
        assert np.array_equal(getattr(runs[0], f), getattr(runs[1], f)), f
