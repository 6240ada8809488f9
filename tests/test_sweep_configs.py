"""Every launch configuration of the window sweep gives the same bits and the
counting sweep's pairs: where candidates lie at the cutoff (four a particle
in 2-D, thirty in 3-D), where chunks and their lists of candidates left over
run full, and where two particles share a place."""
import numpy as np
import pytest

import grasph_b200 as G
from gc_helpers import make_backend
from test_sweep_window import _build, _counts

pytestmark = pytest.mark.gpu


def _run(shape, functor, precision, config, coincident):
    lf = _build(shape, functor, "spline")
    ps = lf.systems[0]
    if coincident:
        ps.x[ps.n // 2] = ps.x[ps.n // 2 + 1]
    s = G.Session([lf], backend=make_backend("cuda"), precision=precision)
    s.backend.set_sweep_config(config)
    s.push()
    si = lf.interactions[0]
    s.sort_particles(ps, 2.0 * si.kernel.h)
    s.create_grid(si)
    for stage in range(1, len(si.pfns) + 1):
        s.sweep(si, stage)
    s.pull()
    return ps


@pytest.mark.parametrize("precision", [G.PRECISION_FP64, G.PRECISION_FP32_COMPENSATED])
@pytest.mark.parametrize("functor", ["fluid", "stress"])
@pytest.mark.parametrize("shape,coincident", [("on_the_cutoff_2d", False), ("on_the_cutoff_3d", False),
                                              ("on_the_cutoff_2d", True), ("chunks_2d", False), ("chunks_3d", True),
                                              ("one_cell", True)])
def test_same_bits(shape, coincident, functor, precision):
    ref = _run(shape, functor, precision, 0, coincident)
    assert np.isnan(ref.drhodt).sum() == (2 if coincident else 0)
    for config in range(1, 4):
        ps = _run(shape, functor, precision, config, coincident)
        for f, _ in ps.particle_fields():
            assert np.array_equal(getattr(ps, f), getattr(ref, f), equal_nan=f != "id"), f"{config} {f}"


@pytest.mark.parametrize("precision", [G.PRECISION_FP64, G.PRECISION_FP32_COMPENSATED])
@pytest.mark.parametrize("config", range(4))
@pytest.mark.parametrize("shape", ["on_the_cutoff_2d", "on_the_cutoff_3d", "chunks_3d"])
def test_pairs(shape, config, precision):
    lf = _build(shape, "stress", "spline")
    s = G.Session([lf], backend=make_backend("cuda"), precision=precision)
    s.backend.set_sweep_config(config)
    s.push()
    s.step(1, 0.01)
    assert s.stats()["pairs_last_step"] == _counts(shape, "stress", "spline").sum() // 2
