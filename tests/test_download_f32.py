"""Float32 systems' fields are rounded to Float32 on the device: the bits of a
Float64 download rounded on the host, for several instances, odd sizes, a
strided array and calls that one staging buffer does not hold."""
import numpy as np
import pytest

import grasph_b200 as G
import grasph_b200.engine as engine
from gc_helpers import make_backend

pytestmark = pytest.mark.gpu


def _column(n, seed):
    T, rng = np.float32, np.random.default_rng(seed)
    ps = G.ElastoPlasticParticleSystem("s", n, 2, 4, T(1.0), T(10.0), dtype=T)
    ps.x[:] = rng.uniform(0.0, 1.0, ps.x.shape)
    ps.v[:] = rng.standard_normal(ps.v.shape)
    ps.rho[:] = 1000.0
    ps.stress[:] = rng.standard_normal(ps.stress.shape)
    h = T(0.1)
    inter = G.SystemInteraction(G.CubicSplineKernel(h, ndims=2),
                                (G.StrainRateVorticityPfn(), G.CauchyFluidPfn(T(0.1), T(0.1), h)), ps)
    return G.LeapFrogTimeIntegrator([ps], [inter])


@pytest.mark.parametrize("limit", [engine.DOWNLOAD_BYTES, 1])
def test_float32_download_is_the_rounded_float64_one(limit, monkeypatch):
    monkeypatch.setattr(engine, "DOWNLOAD_BYTES", limit)
    lfs = [_column(n, n) for n in (1, 37, 260)]
    s = G.Session(lfs, backend=make_backend("cuda"))
    s.push()
    s.step(3, 0.05)
    strided = np.zeros((260, 8), np.float32)
    lfs[2].systems[0].stress = strided[:, ::2]
    s.pull()
    for lf, m in zip(lfs, s.maps):
        ps = lf.systems[0]
        for name, fid in ps.particle_fields():
            a = getattr(ps, name)
            wide = np.zeros(a.shape, np.int64 if name == "id" else np.float64)
            s.backend.download_into(m.inst, m.h(ps), fid, wide)
            assert np.array_equal(a, wide.astype(a.dtype)), name
    assert np.any(strided[:, ::2]) and not np.any(strided[:, 1::2])
