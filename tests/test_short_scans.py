"""Grids and sorts of few cells are scanned by one block.  Two clusters of
water moved apart so that the cells go from one pass of the block over its
second one to the tiled scans: the sorted order and the sums are the
oracle's, in single exact steps and in captured ones."""
import numpy as np
import pytest

import grasph_b200 as G
from gc_helpers import make_backend

pytestmark = pytest.mark.gpu

H, ROWS = 0.06, 20  # the clusters' cells: 0.12 wide, about 20 rows of them


def _clusters(cells):
    rng = np.random.default_rng(cells)
    n, height = 240, ROWS * 2.0 * H
    ps = G.FluidParticleSystem("w", n, 2, 1.0, 20.0, state_updater=G.TaitEOSUpdater(1000.0))
    ps.x[:] = rng.uniform(0.0, 1.0, ps.x.shape) * (0.3, height)
    ps.x[n // 2:, 0] += cells / ROWS * 2.0 * H
    ps.v[:] = rng.standard_normal(ps.v.shape)
    ps.rho[:] = 1000.0
    wall = G.BasicParticleSystem("b", 60, 2, 1.0, 20.0)
    wall.x[:] = rng.uniform(0.0, 1.0, wall.x.shape) * (0.3, height)
    wall.rho[:] = 1000.0
    k, pfn = G.CubicSplineKernel(H, ndims=2), G.FluidPfn(0.1, 0.1, H)
    bound = G.DynamicBoundarySystem(wall, (0.0, 1.0), (0.0, 0.0), 3.0)
    inters = [G.SystemInteraction(k, pfn, ps), G.SystemInteraction(k, pfn, ps, bound)]
    return G.LeapFrogTimeIntegrator([ps, wall], inters), ps


@pytest.mark.parametrize("graphs", [False, True])
@pytest.mark.parametrize("cells", [100, 1000, 6000, 7200, 14000, 15600, 17000, 60000])
def test_scans_of_few_cells(cells, graphs):
    runs = []
    for name in ("cuda", "oracle"):
        lf, ps = _clusters(cells)
        s = G.Session([lf], backend=make_backend(name))
        if name == "cuda":
            s.backend.set_graphs(graphs, 4, 0.0)
        s.push()
        s.step(16, 0.05)
        s.pull()
        runs.append(ps)
    a, b = runs
    assert np.array_equal(a.id, b.id)
    # sums of up to a hundred terms over 16 steps, in 53 bits
    for name, _ in a.particle_fields():
        x, y = getattr(a, name), getattr(b, name)
        assert np.abs(x - y).max() <= 1e-10 * np.abs(y).max(), name
