"""The clustered triangular solve where a CTA keeps only its own blocks of the solution:
many right-hand sides from about 2400 panels, fewer from 2900 (there on both sides of
the line, which odd orders meet earlier), one from about 10,000.  Even and odd
orders, whole and partial last blocks, both directions, clusters of 8 and 7 CTAs, and
a wait that runs out.

Bound: the factors' product is 1/2 on the diagonal and 0.3 / sqrt(n) beside it, so
its condition is below 10 and a row's 2-norm below 1; FP32 substitution with n <= 4200
terms of random sign rounds to within 5e-6 of the largest entry, and a residual adds
entries of random sign: 1e-5 of the largest entry is asked."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _matrices(rng, nb, n):
    a = rng.standard_normal((2, n, n), dtype=np.float32) + 1j * rng.standard_normal((2, n, n), dtype=np.float32)
    a *= np.float32(0.3 / np.sqrt(n))
    a[:, np.arange(n), np.arange(n)] += 0.5
    return a[np.arange(nb) % 2].astype(np.complex128)


@pytest.mark.parametrize("conj", [False, True])
@pytest.mark.parametrize("nb,n,nrhs", [(1, 2400, 8), (2, 2433, 8), (1, 2496, 16), (16, 2400, 7), (1, 4160, 6), (1, 4199, 5),
                                       (1, 2943, 2), (1, 2943, 3), (1, 2946, 3), (1, 2946, 4)])
def test_own_blocks(mh, gpu, conj, nb, n, nrhs):
    rng = np.random.default_rng(n + nrhs)
    A = _matrices(rng, nb, n)
    B = rng.standard_normal((nb, n, nrhs)) + 1j * rng.standard_normal((nb, n, nrhs))
    LU, bad = gpu.lu_factor_lowp(A)
    assert not bad.any()
    X = gpu.lu_solve_lowp(A, B, conj_trans=conj)
    for b in range(0, nb, 5):
        lu = LU[b].astype(np.complex128)
        U, L = np.triu(lu), np.tril(lu, -1)
        if conj:
            Y = U.conj().T @ (X[b] + L.conj().T @ X[b])
        else:
            Y = U @ X[b]
            Y = Y + L @ Y
        assert np.max(np.abs(Y - B[b])) <= 1e-5 * np.max(np.abs(X[b])), b


def test_timeout_is_reported(mh, gpu):
    rng = np.random.default_rng(5)
    A = _matrices(rng, 1, 2400)
    B = rng.standard_normal((1, 2400, 8)) + 0j
    gpu.set_wait_injection(True)
    try:
        with pytest.raises(mh.native.DeviceTimeoutError):
            gpu.lu_solve_lowp(A, B)
    finally:
        gpu.set_wait_injection(False)
    X = gpu.lu_solve_lowp(A, B)
    assert np.max(np.abs(A[0] @ X[0] - B[0])) <= 1e-2 * np.max(np.abs(X))


def test_twenty_thousand_panels(mh, gpu):
    """Refined to 1e-10 with the tensor-core factors, no matrix falling back."""
    mesh = mh.mesh_hemisphere(1.0, (0.0, 0.0, 0.0), (204, 202))
    dofs = [mh.translational_dofs(mesh, "Heave"), mh.translational_dofs(mesh, "Surge")]
    gfs = (mh.Rankine(), mh.RankineReflected(), mh.GFWu())
    A, B, _, _, info = mh.hydro_batch(mesh, [1.1], dofs, green_functions=gfs, ctx=gpu)
    assert info.n_fallback == 0 and info.max_rel_residual <= 1e-10
    # heave and surge of a body of revolution do not couple
    assert abs(A[0, 1, 0]) <= 1e-6 * A[0, 0, 0] and A[0, 0, 0] > 0.0 and B[0, 0, 0] > 0.0
