"""Matrices with entries that are no finite numbers on the FP64 paths that factor with
the library's pivoted LU, whose pivot search must not see them: a NaN comes through
to the outputs, infinite entries are refused, and the context's later calls are what
they were.  Wu's term is not defined above the free surface: a body that rises out of
the water has NaN and infinite entries.  Forward derivatives of the Delhommeau term
there are refused before anything is launched."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nrhs", [(1201, 1), (1300, 3), (40, 800)])
def test_library_solve(mh, gpu, n, nrhs):
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    b = rng.standard_normal((n, nrhs)) + 0j
    one = np.eye(n, dtype=complex)
    good = np.asarray(mh.solve(A, one, b, ctx=gpu))
    for at in ((0, 0), (n // 2, n // 3), (n - 1, n - 1)):
        M = A.copy()
        M[at] = np.nan
        assert np.isnan(np.asarray(mh.solve(M, one, b, ctx=gpu))).all()
        M[at] = np.inf
        with pytest.raises(mh.SingularMatrixError):
            mh.solve(M, one, b, ctx=gpu)
    assert np.array_equal(np.asarray(mh.solve(A, one, b, ctx=gpu)), good)


@pytest.mark.parametrize("precision", ["mixed", "fp64", "fp64_batched"])
def test_body_out_of_the_water(mh, gpu, precision):
    wet = mh.mesh_hemisphere(1.0, (0.0, 0.0, 0.0), (8, 10))
    dry = wet.translated((0.0, 0.0, 0.3))
    om = [0.4, 1.3, 2.2, 0.9, 1.1, 3.0]

    def call(mesh, direct, w=om):
        dofs = [mh.translational_dofs(mesh, "Heave"), mh.translational_dofs(mesh, "Surge")]
        return mh.hydro_batch(mesh, w, dofs, [0.3], green_functions=(mh.Rankine(), mh.RankineReflected(), mh.GFWu()),
                              direct=direct, precision=precision, ctx=gpu)[:4]

    for direct in (True, False):
        good = call(wet, direct)
        for w in ([1.3], om):
            assert np.isnan(call(dry, direct, w)[0]).any()
        for a, b in zip(good, call(wet, direct)):
            assert np.array_equal(a, b)


def _jvp(mh, gpu, mesh, wave, precision):
    rng = np.random.default_rng(1)
    t = mh.MeshTangent(*(rng.standard_normal(a.shape) * 0.1 for a in (mesh.vertices, mesh.centers, mesh.normals)),
                       rng.standard_normal(mesh.nfaces) * 0.01, np.zeros(mesh.nfaces))
    return mh.hydro_batch_jvp(mesh, [1.3], [mh.translational_dofs(mesh, "Heave")], [], t, t_omegas=np.ones(1), ctx=gpu,
                              precision=precision, green_functions=(mh.Rankine(), mh.RankineReflected(), wave))


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_gradients_out_of_the_water(mh, gpu, precision):
    dry = mh.mesh_hemisphere(1.0, (0.0, 0.0, 0.3), (8, 10))
    r = mh.hydro_batch_vjp(dry, [1.3], [mh.translational_dofs(dry, "Heave")], [], np.ones((1, 1, 1)), np.ones((1, 1, 1)),
                           None, None, green_functions=(mh.Rankine(), mh.RankineReflected(), mh.GFWu()),
                           precision=precision, ctx=gpu)
    assert np.isnan(r.added_mass).any()
    assert np.isnan(_jvp(mh, gpu, dry, mh.GFWu(), precision).d_added_mass).any()


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_forward_derivatives_of_delhommeau_above_the_surface_are_refused(mh, gpu, precision):
    dry = mh.mesh_hemisphere(1.0, (0.0, 0.0, 0.3), (8, 10))
    wet = mh.mesh_hemisphere(1.0, (0.0, 0.0, 0.0), (8, 10))
    for mesh in (dry, mh.combine_meshes([wet, dry]), mh.generate_hemisphere(1.0, (0.0, 0.0, 0.3), (8, 10), ctx=gpu),
                 mh.generate_combined([wet, dry], ctx=gpu)):
        with pytest.raises(mh.ArgumentError, match="free surface"):
            _jvp(mh, gpu, mesh, mh.ExactGuevelDelhommeau(), precision)
    low = mh.generate_hemisphere(1.0, (0.0, 0.0, 0.01), (8, 10), ctx=gpu)  # its centres are below
    for mesh in (wet, low):
        assert np.isfinite(_jvp(mh, gpu, mesh, mh.ExactGuevelDelhommeau(), precision).d_added_mass).all()
