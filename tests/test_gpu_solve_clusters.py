"""The clustered triangular solve of the tensor-core factors: every cluster size
(matrices in a batch: 1 and 10 take eight CTAs each, 20 six, 30 four, 60 two, 160
one, never more than a matrix has row blocks), partial and whole last blocks, odd
panel counts (8-byte copies), right-hand sides in one or two passes, both
directions.

Bound: the solve runs in FP32 on factors of a matrix whose condition is below 10;
substitution with n <= 700 terms of random sign rounds to within 2e-6 of the
largest entry, so 1e-5 is asked, as for the other solves of these factors."""
import numpy as np
import pytest


def _matrices(rng, nb, n):
    a = 0.3 / np.sqrt(n) * (rng.standard_normal((1, n, n)) + 1j * rng.standard_normal((1, n, n)))
    return np.broadcast_to(a[0] + 0.5 * np.eye(n), (nb, n, n))


@pytest.mark.gpu
@pytest.mark.parametrize("conj", [False, True])
@pytest.mark.parametrize("nb,n,nrhs", [(1, 64, 1), (1, 65, 3), (1, 700, 5), (10, 577, 2), (20, 390, 8), (20, 449, 9),
                                       (30, 257, 4), (60, 130, 7), (60, 193, 16), (160, 128, 6), (160, 63, 1)])
def test_clustered_solve(mh, gpu, conj, nb, n, nrhs):
    rng = np.random.default_rng(n + nrhs)
    A = _matrices(rng, nb, n)
    B = rng.standard_normal((nb, n, nrhs)) + 1j * rng.standard_normal((nb, n, nrhs))
    LU, bad = gpu.lu_factor_lowp(A[:1])
    assert not bad.any()
    lu = LU[0].astype(np.complex128)
    M = (np.tril(lu, -1) + np.eye(n)) @ np.triu(lu)
    if conj:
        M = M.conj().T
    X = gpu.lu_solve_lowp(A, B, conj_trans=conj)
    ref = np.linalg.solve(M, B.transpose(1, 0, 2).reshape(n, -1)).reshape(n, nb, nrhs).transpose(1, 0, 2)
    assert np.max(np.abs(X - ref)) <= 1e-5 * np.max(np.abs(ref))
