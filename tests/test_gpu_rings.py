"""The frequency-batched Delhommeau passes past the polar patch (the table's
rings R in [2, 4), [4, 8), [8, 16) and the full table beyond), forward and
tangent, against the adaptive quadrature of every pair: panel counts around
the 64-row tiles, frequencies in any order and in more than one launch.

Bound: the rings reproduce the quadrature to 5e-14 and the quadrature itself
stops at 1e-13 of each term; S and D are sums with coefficients below one, the
solve's condition is below 10 and the tangent one order more: 1e-11 and 1e-10
of the largest output are asked (level 0, everything in FP64)."""
import numpy as np
import pytest

CASES = [
    # radius, second body's distance (0: none), resolution, frequencies, largest omega
    (1.9, 0.0, (9, 15), 7, 3.0),     # patch and first ring, 75 panels
    (1.0, 4.0, (8, 8), 16, 3.0),     # up to the second ring, 64 panels
    (2.0, 9.0, (10, 13), 9, 3.0),    # up to the third, 130 panels
    (1.0, 25.0, (4, 7), 12, 3.0),    # outside the rings too, 28 panels
    (0.3, 0.0, (4, 9), 6, 1.0),      # none past the patch
    (1.9, 0.0, (4, 9), 135, 3.0),    # two launches of frequencies
]


def _mesh(mh, radius, gap, resolution):
    m = mh.mesh_hemisphere(radius, (0.0, 0.0, 0.0), resolution)
    return mh.combine_meshes([m, m.translated((gap, 0.3, 0.0))]) if gap else m


def _setup(mh, radius, gap, resolution, nw, top):
    mesh = _mesh(mh, radius, gap, resolution)
    om = np.random.default_rng(nw).permutation(np.linspace(0.3, top, nw))
    dofs = [mh.translational_dofs(mesh, "Heave"), mh.translational_dofs(mesh, "Surge")]
    return mesh, om, dofs, dict(green_functions=(mh.Rankine(), mh.RankineReflected(), mh.ExactGuevelDelhommeau()))


@pytest.fixture
def exact_too(series_fp64):
    def both(call):
        got = call()
        series_fp64.set_delhommeau_method("exact")
        try:
            return got, call()
        finally:
            series_fp64.set_delhommeau_method("table")
    yield series_fp64, both


@pytest.mark.gpu
@pytest.mark.parametrize("direct", [True, False])
@pytest.mark.parametrize("case", CASES)
def test_rings_against_quadrature(mh, exact_too, case, direct):
    gpu, both = exact_too
    mesh, om, dofs, kw = _setup(mh, *case)
    got, want = both(lambda: mh.hydro_batch(mesh, om, dofs, [0.3], precision="fp64_batched", direct=direct, ctx=gpu, **kw))
    for a, b in zip(got[:4], want[:4]):
        assert np.max(np.abs(a - b)) <= 1e-11 * np.max(np.abs(b))


@pytest.mark.gpu
@pytest.mark.parametrize("case", CASES[:5])
def test_ring_tangents_against_quadrature(mh, exact_too, case):
    gpu, both = exact_too
    mesh, om, dofs, kw = _setup(mh, *case)
    rng = np.random.default_rng(1)
    t = mh.MeshTangent(*(rng.standard_normal(a.shape) * 0.1 for a in (mesh.vertices, mesh.centers, mesh.normals)),
                       rng.standard_normal(mesh.nfaces) * 0.01, np.zeros(mesh.nfaces))
    got, want = both(lambda: mh.hydro_batch_jvp(mesh, om, dofs, [0.3], t, t_omegas=np.ones(len(om)), precision="mixed",
                                                tol=1e-13, ctx=gpu, **kw))
    for f in ("d_added_mass", "d_damping", "d_diffraction"):
        a, b = getattr(got, f), getattr(want, f)
        assert np.max(np.abs(a - b)) <= 1e-10 * np.max(np.abs(b))
