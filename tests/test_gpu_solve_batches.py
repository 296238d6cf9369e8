"""The clustered triangular solve on batches of matrices that differ from their
neighbours: every cluster size (as many CTAs per matrix as let all clusters run at
once, 8 for one matrix down to 1 for 160), batches around the sizes at which the
clusters of a size no longer fit, both directions, one to nine right-hand sides.

Bound as in test_gpu_solve_clusters.py: FP32 substitution with factors of a matrix
whose condition is below 10 rounds to within 2e-6 of the largest entry; 1e-5 is
asked.  Another matrix's factors differ by about its off-diagonal part, 0.3."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _batch(rng, nb, n):
    """Five different matrices in turn, no two neighbours (of up to four) alike."""
    a = 0.3 / np.sqrt(n) * (rng.standard_normal((5, n, n)) + 1j * rng.standard_normal((5, n, n)))
    return (a + 0.5 * np.eye(n))[np.arange(nb) % 5]


@pytest.mark.parametrize("conj", [False, True])
@pytest.mark.parametrize("nb,n,nrhs", [(1, 520, 2), (15, 513, 1), (16, 520, 3), (18, 449, 4), (22, 390, 2), (24, 385, 8),
                                       (27, 321, 1), (30, 330, 5), (36, 257, 4), (37, 258, 1), (45, 200, 9), (48, 193, 2),
                                       (74, 130, 3), (75, 131, 2), (160, 130, 1)])
def test_every_matrix_its_own(mh, gpu, conj, nb, n, nrhs):
    rng = np.random.default_rng(nb + n + nrhs)
    A = _batch(rng, nb, n)
    B = rng.standard_normal((nb, n, nrhs)) + 1j * rng.standard_normal((nb, n, nrhs))
    LU, bad = gpu.lu_factor_lowp(A)
    assert not bad.any()
    X = gpu.lu_solve_lowp(A, B, conj_trans=conj)
    for b in range(nb):
        lu = LU[b].astype(np.complex128)
        M = (np.tril(lu, -1) + np.eye(n)) @ np.triu(lu)
        ref = np.linalg.solve(M.conj().T if conj else M, B[b])
        assert np.max(np.abs(X[b] - ref)) <= 1e-5 * np.max(np.abs(ref)), b
