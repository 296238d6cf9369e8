"""Forward-mode derivatives of calls with hundreds and thousands of frequencies:
the tabulated Delhommeau tangents are launched for some of them at a time.

Bounds: against the adaptive quadrature as in test_gpu_rings.py, 1e-10 of the
largest output (both solved to 1e-13).  A call of thousands against two calls of
half its frequencies: every frequency has its own matrices and its own solve to a
relative residual of 1e-10, whose condition is below 10 (no irregular frequency in
the range), and so has its tangent: 1e-8 of the largest output is asked."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _setup(mh, nw):
    one = mh.mesh_hemisphere(1.0, (0.0, 0.0, 0.0), (4, 7))
    mesh = mh.combine_meshes([one, one.translated((7.0, 0.3, 0.0))])  # 28 panels, the patch and all rings
    rng = np.random.default_rng(nw)
    om = rng.permutation(np.linspace(0.3, 3.0, nw))
    t = mh.MeshTangent(*(rng.standard_normal(a.shape) * 0.1 for a in (mesh.vertices, mesh.centers, mesh.normals)),
                       rng.standard_normal(mesh.nfaces) * 0.01, np.zeros(mesh.nfaces))
    gfs = (mh.Rankine(), mh.RankineReflected(), mh.ExactGuevelDelhommeau())
    return mesh, om, [mh.translational_dofs(mesh, "Heave")], t, rng.standard_normal(nw), gfs


def test_windows_against_quadrature(mh, series_fp64):
    gpu = series_fp64
    mesh, om, dofs, t, tw, gfs = _setup(mh, 1026)  # three launches

    def call():
        return mh.hydro_batch_jvp(mesh, om, dofs, [0.3], t, t_omegas=tw, green_functions=gfs, precision="mixed",
                                  tol=1e-13, ctx=gpu)
    got = call()
    gpu.set_delhommeau_method("exact")
    try:
        want = call()
    finally:
        gpu.set_delhommeau_method("table")
    for f in ("d_added_mass", "d_damping", "d_diffraction"):
        a, b = getattr(got, f), getattr(want, f)
        assert np.max(np.abs(a - b)) <= 1e-10 * np.max(np.abs(b))


@pytest.mark.parametrize("nw", [5600, 6200])
def test_thousands_of_frequencies(mh, gpu, nw):
    mesh, om, dofs, t, tw, gfs = _setup(mh, nw)

    def call(s):
        return mh.hydro_batch_jvp(mesh, om[s], dofs, [0.3], t, t_omegas=tw[s], green_functions=gfs, ctx=gpu)
    got, parts = call(slice(None)), [call(slice(0, nw // 2)), call(slice(nw // 2, None))]
    for f, axis in (("added_mass", -1), ("d_added_mass", -1), ("d_damping", -1), ("d_diffraction", 1)):
        a, b = getattr(got, f), np.concatenate([getattr(p, f) for p in parts], axis=axis)
        assert np.max(np.abs(a - b)) <= 1e-8 * np.max(np.abs(b)), f
