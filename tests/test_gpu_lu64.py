"""FP64 solve with partial pivoting (one CTA up to 96 while the right-hand sides fit
its shared memory, else panels): orders on both sides of that line, at the edges of
a panel (16 columns, fewer where the rows are many), of the update's
column blocks (8) and of the back substitution's blocks (32), several right-hand
sides, matrices that need row exchanges at every column.

Tolerance: Gaussian elimination with partial pivoting solves (A + E) x = b with
|E| <= 3 n u |L| |U| (u = 2^-53), |L| <= 1 and max |U| <= g max |A|; the growth g
of random matrices is about n^(2/3).  So max |A x - b| <= 3 n u n g max |A| max |x|
for the full sums; their random signs make it sqrt(n) smaller, not used here."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(A, X, B):
    n = A.shape[0]
    tol = 3 * n * 2.0 ** -53 * n * n ** (2.0 / 3.0) * np.abs(A).max()
    for q in range(B.shape[1]):
        assert np.abs(A @ X[:, q] - B[:, q]).max() <= tol * np.abs(X[:, q]).max()


@pytest.mark.parametrize("n,nrhs", [(1, 1), (2, 3), (7, 1), (8, 2), (15, 1), (16, 1), (17, 2), (31, 1), (32, 9), (33, 1),
                                    (48, 1), (50, 1), (64, 8), (65, 1), (96, 1), (96, 60), (97, 1),
                                    (100, 6), (257, 2), (700, 1), (870, 1),
                                    (896, 3), (1001, 1), (1200, 1), (1201, 1)])
def test_solve(mh, gpu, n, nrhs):
    rng = np.random.default_rng(n + nrhs)
    A = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    A[np.arange(n), np.arange(n)] *= 1e-3  # small diagonal: pivots are elsewhere
    b = rng.standard_normal((n, nrhs)) + 1j * rng.standard_normal((n, nrhs))
    _check(A, np.asarray(mh.solve(A, np.eye(n, dtype=complex), b, ctx=gpu)).reshape(n, nrhs), b)


def test_cyclic_exchanges(mh, gpu):
    """A permuted triangular matrix: every column's pivot is in another row, and
    exact arithmetic gives back the permutation's solution."""
    n = 75
    rng = np.random.default_rng(3)
    U = np.triu(rng.integers(-2, 3, (n, n)).astype(complex), 1) * 2.0 ** -7 + np.eye(n)
    A = np.roll(U, 29, axis=0)
    x = rng.integers(-4, 5, n) + 1j * rng.integers(-4, 5, n)
    X = np.asarray(mh.solve(A, np.eye(n, dtype=complex), A @ x, ctx=gpu)).reshape(n)
    _check(A, X[:, None], (A @ x)[:, None])
    assert np.abs(X - x).max() <= 1e-10
