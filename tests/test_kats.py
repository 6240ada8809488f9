"""Known-answer tests ported from the reference's own test suite.

Each test restates one Grasph.jl test (file:line cited) against a backend:
the CPU oracle always, and libgrasph_cuda.so under the `gpu` marker.  These
pin both implementations to the reference's documented behaviour.
"""
import math

import numpy as np
import pytest

import grasph_b200 as G
from grasph_b200 import consts as C
from gc_helpers import BACKENDS, basic, kernel, keys, lcg_vals, lex_sorted, session


# ------------------------------------------------------------ kernels (CPU)
# test/test_kernels.jl:10-104

def test_kernel_norms_and_shape():
    import pyoracle as O
    cs = C.GC_KERNEL_CUBIC_SPLINE
    assert math.isclose(O.kernel_norm(cs, 1, 1.0), 2 / 3)
    assert math.isclose(O.kernel_norm(cs, 2, 1.0), 10 / (7 * math.pi))
    assert math.isclose(O.kernel_norm(cs, 3, 1.0), 1 / math.pi)
    k = G.CubicSplineKernel(0.1, ndims=2)
    assert math.isclose(k.h, 0.1) and math.isclose(k.interaction_length, 0.2)
    assert O.kernel_norm(cs, 2, 0.1) == k.norm_coeff
    nc = O.kernel_norm(cs, 3, 1.0)
    assert math.isclose(O.kernel_w(cs, 3, 1.0, 0.0), nc * 1.0)
    assert math.isclose(O.kernel_w(cs, 3, 1.0, 1.0), nc * 0.25)
    assert O.kernel_w(cs, 3, 1.0, 2.0) == 0.0
    assert O.kernel_w(cs, 3, 1.0, 2.5) == 0.0 and O.kernel_w(cs, 3, 1.0, 10.0) == 0.0
    for q in np.arange(0.0, 3.0001, 0.1):
        assert O.kernel_w(cs, 3, 1.0, q) >= 0.0
    assert O.kernel_dw_dq(cs, 3, 1.0, 0.0) == 0.0
    assert O.kernel_dw_dq(cs, 3, 1.0, 2.0) == 0.0
    assert O.kernel_dw_dq(cs, 3, 1.0, 3.0) == 0.0
    for q in (0.5, 1.0, 1.5):
        assert O.kernel_dw_dq(cs, 3, 1.0, q) < 0.0


def test_compensated_power_matches_exact_rational():
    import pyoracle as O
    from fractions import Fraction
    rng = np.random.default_rng(5)
    for x in rng.uniform(0.9, 1.1, 200):
        for n in (7, 12, 6, 2, 5):
            exact = Fraction(float(x)) ** n
            got = O.powi(float(x), n)
            # within one ulp of the exact value
            assert abs(Fraction(got) - exact) <= Fraction(math.ulp(float(exact)))


# -------------------------------------------------------------------- sort
# test/test_sorting.jl:50-221

@pytest.mark.parametrize("be", BACKENDS)
def test_sort_row_major_and_arrays_move_together(be):
    ps = basic(n=6)
    pos = np.array([[0.45, 0.05], [0.05, 0.25], [0.25, 0.05], [0.05, 0.05], [0.45, 0.25], [0.25, 0.25]])
    ps.x[:] = pos
    ps.rho[:] = np.arange(1, 7)
    lf, s = session(be, [ps], [G.SystemInteraction(kernel(), None, ps)])
    perm = s.sort_particles(ps, 0.2)
    s.pull()
    assert lex_sorted(keys(ps.x, 0.2))
    for i in range(6):
        assert np.array_equal(ps.x[i], pos[int(ps.rho[i]) - 1])
    assert np.array_equal(ps.id, perm)
    # stable order of the reference: keys (0,0),(0,1),(1,0),(1,1),(2,0),(2,1)
    assert list(perm) == [4, 2, 3, 6, 1, 5]


@pytest.mark.parametrize("be", BACKENDS)
def test_sort_4_particle_case_and_idempotence(be):
    ps = basic(n=4)
    ps.x[:] = [[0.35, 0.05], [0.05, 0.15], [0.25, 0.05], [0.05, 0.05]]
    ps.rho[:] = [1.0, 2.0, 3.0, 4.0]
    orig = ps.x.copy()
    lf, s = session(be, [ps], [G.SystemInteraction(kernel(), None, ps)])
    s.sort_particles(ps, 0.2)
    s.pull()
    assert lex_sorted(keys(ps.x, 0.2))
    for i in range(4):
        assert np.array_equal(ps.x[i], orig[int(ps.rho[i]) - 1])
    first = ps.x.copy()
    perm2 = s.sort_particles(ps, 0.2)
    s.pull()
    assert np.array_equal(ps.x, first)
    assert list(perm2) == [1, 2, 3, 4]


@pytest.mark.parametrize("be", BACKENDS)
def test_sort_already_sorted_and_single_particle(be):
    ps = basic(n=4)
    ps.x[:] = [[0.05, 0.05], [0.05, 0.25], [0.25, 0.05], [0.45, 0.35]]
    expect = ps.x.copy()
    one = basic(n=1)
    one.x[0] = [0.5, 0.5]
    one.rho[0] = 42.0
    lf, s = session(be, [ps, one], [G.SystemInteraction(kernel(), None, ps)])
    assert list(s.sort_particles(ps, 0.2)) == [1, 2, 3, 4]
    s.sort_particles(one, 0.2)
    s.pull()
    assert np.array_equal(ps.x, expect)
    assert one.rho[0] == 42.0 and np.array_equal(one.x[0], [0.5, 0.5])


@pytest.mark.parametrize("be", BACKENDS)
def test_sort_negative_coordinates(be):
    ps = basic(n=3)
    ps.x[:] = [[0.05, 0.05], [-0.15, -0.15], [-0.35, 0.05]]
    ps.rho[:] = [1, 2, 3]
    lf, s = session(be, [ps], [G.SystemInteraction(kernel(), None, ps)])
    s.sort_particles(ps, 0.2)
    s.pull()
    assert lex_sorted(keys(ps.x, 0.2))
    assert list(ps.rho) == [3.0, 2.0, 1.0]


@pytest.mark.parametrize("be", BACKENDS)
def test_sort_3d_row_major(be):
    ps = basic(n=4, nd=3)
    ps.x[:] = [[0.25, 0.05, 0.05], [0.05, 0.25, 0.05], [0.05, 0.05, 0.25], [0.05, 0.05, 0.05]]
    ps.rho[:] = [1, 2, 3, 4]
    lf, s = session(be, [ps], [G.SystemInteraction(kernel(nd=3), None, ps)])
    s.sort_particles(ps, 0.2)
    s.pull()
    k = keys(ps.x, 0.2)
    assert k.tolist() == [[0, 0, 0], [0, 0, 1], [0, 1, 0], [1, 0, 0]]
    assert list(ps.rho) == [4.0, 3.0, 2.0, 1.0]


@pytest.mark.parametrize("be", BACKENDS)
def test_sort_all_fields_of_elastoplastic_move(be):
    n = 50
    rng = np.random.default_rng(3)
    ps = G.ElastoPlasticParticleSystem("ep", n, 2, 4, 1.0, 10.0)
    ps.x[:] = rng.uniform(-1, 1, (n, 2))
    for name in ("v", "rho", "dvdt", "drhodt", "p", "stress", "strain_rate", "vorticity", "strain", "strain_p"):
        a = getattr(ps, name)
        a[...] = rng.normal(size=a.shape)
    before = {name: getattr(ps, name).copy() for name, _ in ps.particle_fields()}
    lf, s = session(be, [ps], [G.SystemInteraction(kernel(), None, ps)])
    perm = s.sort_particles(ps, 0.2) - 1
    s.pull()
    for name, arr in before.items():
        assert np.array_equal(getattr(ps, name), arr[perm]), name
    k = keys(before["x"], 0.2)
    order = sorted(range(n), key=lambda i: (tuple(k[i]), i))
    assert list(perm) == order


# ------------------------------------------------------------------ ghosts
# test/test_sorting.jl:227-334, test/test_ghost_particles.jl:112-193,263-287,
# test/test_ghost_updates.jl:21-52, test/test_ghost_copier.jl:186-304

def _granular(n, ns=3):
    ps = G.StressParticleSystem("g", n, 2, ns, 1.0, 20.0)
    ps.rho[:] = 1850.0
    return ps


@pytest.mark.parametrize("be", BACKENDS)
def test_ghost_generate_mirrors_and_kinematics(be):
    ps = _granular(3)
    ps.x[:] = [[0.3, 0.05], [0.3, 0.20], [0.3, -0.05]]
    ps.v[0] = [1.0, -0.5]
    g = G.GhostParticleSystem(ps, G.GhostCopier("rho"))
    ge = G.GhostEntry(g, 0.15, ((0.0, 1.0), (0.0, 0.0)))
    lf, s = session(be, [ps], [G.SystemInteraction(kernel(), None, ps)], ghosts=[ge])
    s.generate_ghosts(ge)
    s.update_ghost_kinematics(ge)
    s.update_ghost(ge, 1)
    s.pull_ghost(ge)
    assert g.n == 1
    assert np.allclose(g.x[0], [0.3, -0.05])
    n = np.array([0.0, 1.0])
    assert np.allclose(g.v[0], ps.v[0] - 2 * np.dot(ps.v[0], n) * n)
    assert g.rho[0] == ps.rho[0]
    assert g.idx_original[0] == 1


@pytest.mark.parametrize("be", BACKENDS)
def test_ghost_counts_resize(be):
    ps = _granular(4)
    ps.x[:] = [[0.0, 0.05], [0.0, 0.08], [0.0, -0.1], [0.0, 0.5]]
    g = G.GhostParticleSystem(ps)
    ge = G.GhostEntry(g, 0.15, ((0.0, 1.0), (0.0, 0.0)))
    lf, s = session(be, [ps], [G.SystemInteraction(kernel(), None, ps)], ghosts=[ge])
    s.generate_ghosts(ge)
    s.pull_ghost(ge)
    assert g.n == 2
    ps.x[1] = [0.0, 0.5]
    s.push()
    s.generate_ghosts(ge)
    s.pull_ghost(ge)
    assert g.n == 1
    ps.x[1] = [0.0, 0.08]
    ps.x[2] = [0.0, 0.06]
    s.push()
    s.generate_ghosts(ge)
    s.pull_ghost(ge)
    assert g.n == 3
    # none qualify
    ps.x[:] = [[0.0, -0.1], [0.0, -0.2], [0.0, 0.5], [0.0, 0.6]]
    s.push()
    s.generate_ghosts(ge)
    s.pull_ghost(ge)
    assert g.n == 0


@pytest.mark.parametrize("be", BACKENDS)
def test_ghost_idx_boundary_and_sort(be):
    ps = _granular(4)
    ps.x[:] = [[0.05, 0.5], [0.5, 0.05], [0.5, 0.5], [0.05, 0.05]]
    g = G.GhostParticleSystem(ps)
    ge = G.GhostEntry(g, 0.15, ((1.0, 0.0), (0.0, 0.0)), ((0.0, 1.0), (0.0, 0.0)))
    lf, s = session(be, [ps], [G.SystemInteraction(kernel(), None, ps)], ghosts=[ge])
    s.generate_ghosts(ge)
    s.pull_ghost(ge)
    assert g.n == 4
    # generation order: boundary-major, then source index
    assert list(g.idx_boundary) == [1, 1, 2, 2]
    assert list(g.idx_original) == [1, 4, 2, 4]
    for k in range(g.n):
        if g.idx_boundary[k] == 1:
            assert g.x[k][0] < 0
        else:
            assert g.x[k][1] < 0
    pre = {(tuple(g.x[k]), g.idx_original[k], g.idx_boundary[k]) for k in range(g.n)}
    normals_pre = g.normals.copy()
    s.sort_particles(g, 0.1)
    s.pull_ghost(ge)
    post = {(tuple(g.x[k]), g.idx_original[k], g.idx_boundary[k]) for k in range(g.n)}
    assert pre == post
    assert lex_sorted(keys(g.x, 0.1))
    # cached normals are not in the permuted-array list (src/Sorting.jl:33-40)
    assert np.array_equal(g.normals, normals_pre)


@pytest.mark.parametrize("be", BACKENDS)
def test_ghost_sort_two_boundaries_reverses_order(be):
    ps = basic(n=2)
    ps.x[:] = [[0.92, 0.5], [0.05, 0.06]]
    ps.rho[:] = 1000.0
    g = G.GhostParticleSystem(ps)
    ge = G.GhostEntry(g, 0.1, ((-1.0, 0.0), (1.0, 0.0)), ((0.0, 1.0), (0.0, 0.0)))
    lf, s = session(be, [ps], [G.SystemInteraction(kernel(), None, ps)], ghosts=[ge])
    s.generate_ghosts(ge)
    s.sort_particles(g, 0.1)
    s.pull_ghost(ge)
    assert g.n == 2
    for k in range(2):
        nrm, pt = ge.boundaries[g.idx_boundary[k] - 1]
        src = ps.x[g.idx_original[k] - 1]
        da = np.dot(src - pt, nrm)
        assert np.allclose(g.x[k], src - 2 * da * nrm)
    assert list(g.idx_boundary) == [2, 1]


@pytest.mark.parametrize("be", BACKENDS)
@pytest.mark.parametrize("case", ["floor4", "floor3", "diag45", "multi"])
def test_ghost_householder(be, case):
    if case == "floor3":
        ps = _granular(1, ns=3)
        ps.x[0] = [0.1, 0.04]
        ps.stress[0] = [10.0, -5.0, 3.0]
        planes = [((0.0, 1.0), (0.0, 0.0))]
        cutoff = 0.15
    elif case == "diag45":
        ps = _granular(1, ns=4)
        ps.x[0] = [0.05, 0.05]
        ps.stress[0] = [10.0, 20.0, 30.0, 7.0]
        r = 1.0 / math.sqrt(2.0)
        planes = [((r, r), (0.0, 0.0))]
        cutoff = 0.2
    elif case == "multi":
        ps = _granular(2, ns=4)
        ps.x[:] = [[0.04, 0.20], [0.20, 0.04]]
        ps.stress[:] = [[1.0, 2.0, 3.0, 4.0], [5.0, 6.0, 7.0, 8.0]]
        planes = [((1.0, 0.0), (0.0, 0.0)), ((0.0, 1.0), (0.0, 0.0))]
        cutoff = 0.15
    else:
        ps = _granular(2, ns=4)
        ps.x[:] = [[0.1, 0.04], [0.2, 0.06]]
        ps.stress[:] = [[10.0, 20.0, 30.0, 5.0], [-5.0, -5.0, 0.0, -3.0]]
        planes = [((0.0, 1.0), (0.0, 0.0))]
        cutoff = 0.15
    g = G.GhostParticleSystem(ps, G.GhostCopier(("stress", G.HouseholderReflect())))
    ge = G.GhostEntry(g, cutoff, *planes)
    lf, s = session(be, [ps], [G.SystemInteraction(kernel(), None, ps)], ghosts=[ge])
    s.generate_ghosts(ge)
    s.update_ghost(ge, 1)
    s.pull_ghost(ge)
    for k in range(g.n):
        src = ps.stress[g.idx_original[k] - 1]
        if case == "floor3":
            expect = [src[0], src[1], -src[2]]
        elif case == "diag45":
            expect = [20.0, 10.0, 30.0, 7.0]
        else:
            expect = [src[0], src[1], src[2], -src[3]]
        assert np.allclose(g.stress[k], expect, rtol=1e-12, atol=1e-12)


# -------------------------------------------------------------------- grid
# test/test_interaction_grid.jl:46-287, test/test_sorting.jl:340-367

def _cells_of(cs):
    out = {}
    for c in range(1, len(cs)):
        for j in range(cs[c - 1], cs[c]):
            out[j] = c
    return out


@pytest.mark.parametrize("be", BACKENDS)
def test_grid_self_clusters_and_origin(be):
    ps = basic(n=6)
    ps.x[:] = [[0.05, 0.05], [0.06, 0.08], [0.07, 0.06], [0.35, 0.05], [0.36, 0.08], [0.37, 0.06]]
    si = G.SystemInteraction(kernel(), None, ps)
    lf, s = session(be, [ps], [si])
    cs, ming, ng = s.create_grid(si)
    assert cs[-1] - 1 == 6
    cells = _cells_of(cs)
    assert cells[1] == cells[2] == cells[3] and cells[4] == cells[5] == cells[6] and cells[1] != cells[4]
    assert cs[cells[1]] - cs[cells[1] - 1] == 3
    cutoff = 0.2
    raw_min = ps.x.min(axis=0) - 2 * cutoff
    assert np.all(ming <= raw_min + 1e-10)
    for v in ming:
        r = math.fmod(v, cutoff)
        assert abs(r) < 1e-9 or abs(abs(r) - cutoff) < 1e-9
    cs2, ming2, ng2 = s.create_grid(si)
    assert np.array_equal(cs, cs2)


@pytest.mark.parametrize("be", BACKENDS)
def test_grid_coupled(be):
    a = basic(n=3)
    b = basic(n=3)
    a.x[:] = [[0.05, 0.05], [0.06, 0.08], [0.07, 0.06]]
    b.x[:] = [[0.35, 0.05], [0.36, 0.08], [0.37, 0.06]]
    si = G.SystemInteraction(kernel(), None, a, b)
    lf, s = session(be, [a, b], [si])
    cs, ming, ng = s.create_grid(si)
    assert cs[-1] - 1 == 3
    occupied = [c for c in range(1, len(cs)) if cs[c] - cs[c - 1] > 0]
    assert len(occupied) == 1 and cs[occupied[0]] - cs[occupied[0] - 1] == 3
    combined = np.minimum(a.x.min(0), b.x.min(0))
    assert np.all(ming <= combined - 0.4 + 1e-10)


@pytest.mark.parametrize("be", BACKENDS)
def test_grid_alignment_across_interactions(be):
    a = basic(n=4)
    b = basic(n=4)
    a.x[:] = [[0.05, 0.05], [0.07, 0.07], [0.09, 0.05], [0.06, 0.09]]
    b.x[:] = [[0.53, 0.53], [0.55, 0.57], [0.57, 0.55], [0.54, 0.56]]
    sa = G.SystemInteraction(kernel(), None, a)
    sb = G.SystemInteraction(kernel(), None, b)
    lf, s = session(be, [a, b], [sa, sb])
    _, ma, _ = s.create_grid(sa)
    _, mb, _ = s.create_grid(sb)
    d = (ma - mb) / 0.2
    assert np.allclose(d, np.round(d), atol=1e-9)


@pytest.mark.parametrize("be", BACKENDS)
def test_sorted_csr_ranges_map_to_their_cell(be):
    ps = basic(n=12)
    ps.x[0:4] = [[0.05 + i * 0.01, 0.05] for i in range(4)]
    ps.x[4:8] = [[0.45 + i * 0.01, 0.05] for i in range(4)]
    ps.x[8:12] = [[0.05 + i * 0.01, 0.45] for i in range(4)]
    si = G.SystemInteraction(kernel(), None, ps)
    lf, s = session(be, [ps], [si])
    s.sort_particles(ps, 0.2)
    cs, ming, ng = s.create_grid(si)
    s.pull()
    for c in range(1, len(cs)):
        for j in range(cs[c - 1], cs[c]):
            cell = np.floor((ps.x[j - 1] - ming) / 0.2).astype(np.int64)
            assert cell[0] * ng[1] + cell[1] + 1 == c


# ---------------------------------------------------- sweep pair counting
# test/test_interaction_sweep.jl:170-209,311-355,408-443,
# test/test_interaction_sweep_3d.jl:109-147

def _count_sweep(be, systems, inters, stage_inters):
    lf, s = session(be, systems, inters)
    for si in stage_inters:
        s.create_grid(si)
        s.sweep(si, 1)
    s.pull()
    return s


@pytest.mark.parametrize("be", BACKENDS)
def test_self_sweep_counts(be):
    ps = basic(n=3)
    ps.x[:] = [[0.05, 0.05], [0.10, 0.10], [0.25, 0.25]]
    si = G.SystemInteraction(kernel(), G.CountingPfn(), ps)
    _count_sweep(be, [ps], [si], [si])
    assert list(ps.dvdt[:, 0]) == [1.0, 1.0, 0.0]
    assert list(ps.drhodt) == [1.0, 1.0, 0.0]


@pytest.mark.parametrize("be", BACKENDS)
def test_self_sweep_8_all_within(be):
    ps = basic(n=8)
    v = lcg_vals(16)
    ps.x[:] = np.array(v).reshape(8, 2)
    si = G.SystemInteraction(kernel(), G.CountingPfn(), ps)
    _count_sweep(be, [ps], [si], [si])
    assert np.all(ps.dvdt[:, 0] == 7.0) and np.all(ps.drhodt == 7.0)


@pytest.mark.parametrize("be", BACKENDS)
def test_self_sweep_far_pair(be):
    ps = basic(n=2)
    ps.x[:] = [[0.0, 0.0], [1.0, 1.0]]
    si = G.SystemInteraction(kernel(), G.CountingPfn(), ps)
    _count_sweep(be, [ps], [si], [si])
    assert np.all(ps.dvdt == 0.0) and np.all(ps.drhodt == 0.0)


@pytest.mark.parametrize("be", BACKENDS)
def test_coupled_sweep_counts(be):
    a = basic(n=3)
    b = basic(n=3)
    a.x[:] = [[0.05, 0.05], [0.10, 0.10], [0.50, 0.50]]
    b.x[:] = [[0.06, 0.06], [0.11, 0.11], [0.55, 0.55]]
    si = G.SystemInteraction(kernel(), G.CountingPfn(), a, b)
    _count_sweep(be, [a, b], [si], [si])
    assert list(a.dvdt[:, 0]) == [2.0, 2.0, 1.0] and list(a.drhodt) == [2.0, 2.0, 1.0]
    assert list(b.dvdt[:, 0]) == [2.0, 2.0, 1.0] and list(b.drhodt) == [2.0, 2.0, 1.0]


@pytest.mark.parametrize("be", BACKENDS)
def test_coupled_sweep_8_each(be):
    a = basic(n=8)
    b = basic(n=8)
    a.x[:] = np.array(lcg_vals(16)).reshape(8, 2)
    b.x[:] = np.array(lcg_vals(16, offset=16)).reshape(8, 2)
    si = G.SystemInteraction(kernel(), G.CountingPfn(), a, b)
    _count_sweep(be, [a, b], [si], [si])
    assert np.all(a.dvdt[:, 0] == 8.0) and np.all(b.dvdt[:, 0] == 8.0)


@pytest.mark.parametrize("be", BACKENDS)
def test_two_interactions_accumulate(be):
    a = basic(n=2)
    b = basic(n=1)
    a.x[:] = [[0.05, 0.05], [0.10, 0.10]]
    b.x[:] = [[0.07, 0.07]]
    s1 = G.SystemInteraction(kernel(), G.CountingPfn(), a)
    s2 = G.SystemInteraction(kernel(), G.CountingPfn(), a, b)
    _count_sweep(be, [a, b], [s1, s2], [s1, s2])
    assert list(a.dvdt[:, 0]) == [2.0, 2.0] and list(a.drhodt) == [2.0, 2.0]
    assert list(b.dvdt[:, 0]) == [2.0] and list(b.drhodt) == [2.0]


@pytest.mark.parametrize("be", BACKENDS)
def test_sweep_3d_counts(be):
    ps = basic(n=3, nd=3)
    ps.x[:] = [[0.05, 0.05, 0.05], [0.10, 0.10, 0.10], [0.50, 0.50, 0.50]]
    si = G.SystemInteraction(kernel(nd=3), G.CountingPfn(), ps)
    _count_sweep(be, [ps], [si], [si])
    assert list(ps.dvdt[:, 0]) == [1.0, 1.0, 0.0]
    a = basic(n=2, nd=3)
    b = basic(n=2, nd=3)
    a.x[:] = [[0.05, 0.05, 0.05], [0.50, 0.50, 0.50]]
    b.x[:] = [[0.06, 0.06, 0.06], [0.51, 0.51, 0.51]]
    sc = G.SystemInteraction(kernel(nd=3), G.CountingPfn(), a, b)
    _count_sweep(be, [a, b], [sc], [sc])
    assert list(a.dvdt[:, 0]) == [1.0, 1.0] and list(b.dvdt[:, 0]) == [1.0, 1.0]


# ------------------------------------------------------------ EP updater
# test/test_ep_updater.jl:18-85

def _ep_one():
    return G.ElastoPlasticParticleSystem("t", 1, 2, 4, 1.0, 100.0)


@pytest.mark.parametrize("be", BACKENDS)
def test_ep_elastic_jaumann_plastic(be):
    E, nu, phi, psi, dt = 1.0e6, 0.3, 30.0 * math.pi / 180.0, 0.0, 0.001
    # elastic increment
    ps = _ep_one()
    ps.strain_rate[0] = [0.1, 0.0, 0.0, 0.0]
    ps.state_updater = (G.ElastoPlasticStressUpdater(E, nu, phi, psi, 1.0e6),)
    lf, s = session(be, [ps], [G.SystemInteraction(kernel(), None, ps)])
    s.update_state(ps, 1, dt)
    s.pull()
    D0 = E / ((1 + nu) * (1 - 2 * nu))
    de = 0.1 * dt
    assert math.isclose(ps.stress[0][0], D0 * (1 - nu) * de)
    assert math.isclose(ps.stress[0][1], D0 * nu * de)
    assert math.isclose(ps.stress[0][2], D0 * nu * de)
    assert ps.stress[0][3] == 0.0
    assert np.allclose(ps.strain[0], ps.strain_rate[0] * dt)
    assert np.all(ps.strain_p[0] == 0.0)
    # Jaumann rotation
    ps = _ep_one()
    ps.stress[0] = [1.0e5, 0.0, 0.0, 0.0]
    ps.vorticity[0] = 10.0
    ps.state_updater = (G.ElastoPlasticStressUpdater(E, nu, phi, psi, 1.0e6),)
    lf, s = session(be, [ps], [G.SystemInteraction(kernel(), None, ps)])
    s.update_state(ps, 1, dt)
    s.pull()
    assert math.isclose(ps.stress[0][3], 1000.0) and math.isclose(ps.stress[0][0], 1.0e5)
    # plastic return lands on the yield surface
    ps = _ep_one()
    ps.strain_rate[0] = [0.0, 0.0, 0.0, 100.0]
    ps.state_updater = (G.ElastoPlasticStressUpdater(E, nu, phi, psi, 10.0),)
    lf, s = session(be, [ps], [G.SystemInteraction(kernel(), None, ps)])
    s.update_state(ps, 1, dt)
    s.pull()
    a_phi = 2 * math.sin(phi) / (math.sqrt(3) * (3 - math.sin(phi)))
    k_c = 6 * 10.0 * math.cos(phi) / (math.sqrt(3) * (3 - math.sin(phi)))
    sig = ps.stress[0]
    I1 = sig[0] + sig[1] + sig[2]
    sd = [sig[0] - I1 / 3, sig[1] - I1 / 3, sig[2] - I1 / 3]
    J2 = 0.5 * (sd[0] ** 2 + sd[1] ** 2 + sd[2] ** 2 + 2 * sig[3] ** 2)
    assert abs(a_phi * I1 + math.sqrt(J2) - k_c) <= 1e-7
    assert np.any(ps.strain_p[0] != 0.0)


# ------------------------------------------------------------- vorticity
# test/test_vorticity.jl:45-84

@pytest.mark.parametrize("be", BACKENDS)
def test_strain_rate_vorticity_pair(be):
    h, rho0 = 0.1, 1000.0
    mass = rho0 * h * h
    ps = G.ElastoPlasticParticleSystem("t", 2, 2, 4, mass, 10.0)
    ps.x[:] = [[0.0, 0.0], [0.05, 0.0]]
    ps.v[:] = [[0.0, 0.0], [0.0, 1.0]]
    ps.rho[:] = rho0
    si = G.SystemInteraction(G.CubicSplineKernel(h, ndims=2), G.StrainRateVorticityPfn(), ps)
    lf, s = session(be, [ps], [si])
    s.create_grid(si)
    s.sweep(si, 1)
    s.pull()
    assert np.any(ps.strain_rate[0] != 0) and np.any(ps.strain_rate[1] != 0)
    k = G.CubicSplineKernel(h, ndims=2)
    dx = ps.x[0] - ps.x[1]
    r = np.linalg.norm(dx)
    q = r / h
    a, b = max(0.0, 2 - q), max(0.0, 1 - q)
    dwdq = k.norm_coeff * (-3.0 * (0.25 * a * a - b * b))
    gx = dwdq * dx / (r * h)
    dv = ps.v[1] - ps.v[0]
    vor = 0.5 * (dv[0] * gx[1] - dv[1] * gx[0]) * (mass / rho0)
    assert math.isclose(ps.vorticity[0], vor, rel_tol=1e-12)
    assert math.isclose(ps.vorticity[1], vor, rel_tol=1e-12)


# ----------------------------------------------------------- integration
# test/test_time_integration.jl:81-195

@pytest.mark.parametrize("be", BACKENDS)
def test_integrator_kinematics(be):
    # constant velocity advances x by 3 dt
    ps = basic(n=1, c=10.0)
    ps.v[0] = [1.0, 0.0]
    ps.rho[:] = 1000.0
    lf, s = session(be, [ps], [G.SystemInteraction(kernel(), None, ps)])
    s.step(3, 0.5)
    s.pull()
    dt = 0.5 * 0.1 / 10.0
    assert abs(ps.x[0][0] - 3 * dt) <= 1e-10 and abs(ps.x[0][1]) <= 1e-10
    # zero velocity keeps x; zero source keeps rho
    ps = basic(n=2, c=10.0)
    ps.x[:] = [[0.2, 0.2], [0.4, 0.4]]
    ps.rho[:] = [800.0, 1200.0]
    x0 = ps.x.copy()
    lf, s = session(be, [ps], [G.SystemInteraction(kernel(), None, ps)])
    s.step(5, 0.5)
    s.pull()
    assert np.allclose(ps.x, x0, atol=1e-12) and np.allclose(ps.rho, [800.0, 1200.0], atol=1e-12)
    # source_v drives the particle down, and dvdt is reset to the source
    ps = basic(n=1, c=10.0, source_v=[0.0, -1.0])
    ps.x[0] = [0.5, 0.5]
    ps.rho[:] = 1000.0
    lf, s = session(be, [ps], [G.SystemInteraction(kernel(), None, ps)])
    s.step(4, 0.5)
    s.pull()
    assert ps.v[0][1] < 0 and ps.x[0][1] < 0.5 and abs(ps.v[0][0]) <= 1e-12
    assert np.array_equal(ps.dvdt[0], [0.0, -1.0])


@pytest.mark.parametrize("be", BACKENDS)
def test_integrator_regenerates_ghosts_and_mirrors_stress(be):
    # test/test_ghost_particles.jl:289-318
    ps = _granular(2)
    ps.x[:] = [[0.0, 0.04], [0.0, 0.03]]
    ps.v[:] = [[0.5, 0.0], [0.0, 0.0]]
    ps.stress[:] = [[1.0, 2.0, 3.0], [4.0, 5.0, 6.0]]
    g = G.GhostParticleSystem(ps, G.GhostCopier("rho", "stress"))
    ge = G.GhostEntry(g, 0.15, ((0.0, 1.0), (0.0, 0.0)))
    si = G.SystemInteraction(G.CubicSplineKernel(0.1, ndims=2), G.StrainRatePfn(), ps, g)
    lf, s = session(be, [ps], [si], ghosts=[ge])
    s.step(1, 0.1)
    s.pull()
    assert g.n == 2
    for k in range(g.n):
        assert np.array_equal(g.stress[k], ps.stress[g.idx_original[k] - 1])
    assert np.any(ps.strain_rate != 0.0)


# ------------------------------------------------ visco-plastic Mohr–Coulomb
# src/StateUpdaters.jl:144-186.  No reference test pins it; the expected
# values restate its formula for two strain-rate states: inside the yield
# cone (stress along the strain rate, minus p) and past the apex (zero).

@pytest.mark.parametrize("be", BACKENDS)
def test_viscoplastic_mc_updater(be):
    rho0, phi, coh = 1850.0, 0.35, 50.0
    ps = G.StressParticleSystem("s", 2, 2, 3, 1.0, 20.0, state_updater=(
        G.ViscoPlasticMCStressUpdater(G.LinearEOSUpdater(rho0), phi, coh),))
    ps.x[:] = [[0.0, 0.0], [1.0, 1.0]]
    ps.rho[:] = [1851.0, 1849.0]
    ps.strain_rate[:] = [[-0.3, 0.1, 0.05], [0.2, 0.3, -0.1]]
    lf, s = session(be, [ps], [G.SystemInteraction(kernel(), None, ps)])
    s.update_state(ps, 1, 1e-4)
    s.pull()
    for i in range(2):
        p = 20.0 * 20.0 * (ps.rho[i] - rho0)
        sr = ps.strain_rate[i]
        m = max(math.sqrt(sr[0] * sr[0] + sr[1] * sr[1] + 2.0 * (sr[2] * sr[2])), 2.220446049250313e-16)
        sc = 2.0 * (coh + p * math.tan(phi))
        st = [(sc * sr[q]) / m - (p if q < 2 else 0.0) for q in range(3)]
        if st[0] + st[1] > 0.0:
            st = [0.0, 0.0, 0.0]
        assert ps.p[i] == p
        assert list(ps.stress[i]) == st


# ---------------------------------------- static (Lennard-Jones) boundary
# FluidPfn against a StaticBoundarySystem, src/PairwiseFunctors.jl:209-219:
# dv/dt_i += -m_j·Π_ij·∇W + f_LJ·dx with artificial_viscosity
# (src/PairwisePhysics.jl:29-34) and lennard_jones(dx, lj_cutoff, c_a, 12, 6)
# (:258-263); the density rate is untouched.

def _lj_expected(xi, xj, vi, vj, rho_i, rho_j, m_j, c, h, alpha, beta, cut):
    dx = np.asarray(xi, float) - np.asarray(xj, float)
    dv = np.asarray(vi, float) - np.asarray(vj, float)
    rr = float(dx @ dx)
    r = math.sqrt(rr)
    q = r / h
    nd = dx.size
    norm = 10.0 / (7.0 * math.pi * h * h) if nd == 2 else 1.0 / (math.pi * h ** 3)
    dwdq = norm * (-3.0 * (0.25 * max(0.0, 2.0 - q) ** 2 - max(0.0, 1.0 - q) ** 2))
    gx = dwdq / (r * h) * dx
    vr = min(float(dx @ dv), 0.0)
    muv = h * vr / (rr + h * h * 0.01)
    piv = (beta * muv - alpha * c) * muv / (0.5 * rho_i * rho_j)
    f = ((cut / r) ** 12 - (cut / r) ** 6) / rr if r < cut else 0.0
    return -m_j * piv * gx + 0.01 * c * c * f * dx


@pytest.mark.parametrize("be", BACKENDS)
@pytest.mark.parametrize("nd", [2, 3])
@pytest.mark.parametrize("sep", [0.8, 1.0, 1.6])
def test_static_boundary_lennard_jones_pair(be, nd, sep):
    """One fluid particle moving towards one static wall particle at
    sep·lj_cutoff: inside the cutoff LJ repulsion plus viscosity; at exactly
    the cutoff and beyond (still inside 2h) viscosity alone."""
    dx_sp, h, c, alpha, beta = 0.5, 0.6, 20.0, 0.3, 0.2
    f = G.FluidParticleSystem("fluid", 1, nd, 250.0, c)
    w = G.BasicParticleSystem("wall", 1, nd, 125.0, c)
    f.x[0] = [0.1] * (nd - 1) + [sep * dx_sp]
    w.x[0] = [0.1] * nd
    w.x[0, -1] = 0.0
    f.v[0] = [0.3] + [0.0] * (nd - 2) + [-1.5]
    f.rho[:] = 1003.0
    w.rho[:] = 998.0
    f.p[:] = 1234.0
    si = G.SystemInteraction(G.CubicSplineKernel(h, ndims=nd), G.FluidPfn(alpha, beta, h), f,
                             G.StaticBoundarySystem(w, dx_sp))
    lf, s = session(be, [f, w], [si])
    s.create_grid(si)
    s.sweep(si, 1)
    s.pull()
    want = _lj_expected(f.x[0], w.x[0], f.v[0], w.v[0], 1003.0, 998.0, 125.0, c, h, alpha, beta, dx_sp)
    assert np.allclose(f.dvdt[0], want, rtol=1e-13, atol=0.0), (f.dvdt[0], want)
    assert f.drhodt[0] == 0.0
    assert np.all(w.dvdt == 0.0) and w.drhodt[0] == 0.0
    if sep < 1.0:
        # the repulsion points away from the wall and dominates
        assert f.dvdt[0, -1] > 0.0


@pytest.mark.parametrize("be", BACKENDS)
@pytest.mark.parametrize("nd", [2, 3])
def test_static_boundary_without_mass(be, nd):
    """A wall's mass scales its viscosity alone: without one the repulsion stays."""
    h, c, dx_sp = 0.6, 30.0, 0.5
    f = G.FluidParticleSystem("f", 1, nd, 125.0, c)
    w = G.BasicParticleSystem("w", 1, nd, 0.0, c)
    f.x[0] = [0.1] * (nd - 1) + [0.4]
    w.x[0] = [0.0] * nd
    f.v[0, -1] = -0.3
    f.rho[:] = 1003.0
    w.rho[:] = 998.0
    si = G.SystemInteraction(G.CubicSplineKernel(h, ndims=nd), G.FluidPfn(0.1, 0.2, h), f,
                             G.StaticBoundarySystem(w, dx_sp))
    lf, s = session(be, [f, w], [si])
    s.create_grid(si)
    s.sweep(si, 1)
    s.pull()
    want = _lj_expected(f.x[0], w.x[0], f.v[0], w.v[0], 1003.0, 998.0, 0.0, c, h, 0.1, 0.2, dx_sp)
    assert want[-1] > 0.0
    assert np.allclose(f.dvdt[0], want, rtol=1e-13, atol=0.0), (f.dvdt[0], want)
