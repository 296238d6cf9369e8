"""The FP64 pivoted solve's choice of pivots and of its kernels: one CTA and panels
on both sides of their line (by order and right-hand sides), panels and the library on
theirs (768 right-hand sides, 1200 rows), whole and ragged panels and blocks.

test_residual's bound separates elimination with and without exchanges: for these
matrices (small diagonal) max |A x - b| / (n u max |A| max |x|), u = 2^-53, is 0.3 to
2 in numpy's arithmetic with the pivots of largest |re| + |im| (n 16 to 700, growing
as n^(1/2)), 40 to 490 without exchanges; 8 is asked.

The permuted triangular matrices have one pivot of size 1 per column, in another row
each time, and entries below 2^-6 else: any other choice grows by 2^6 a column and
overflows.  Their entries and solutions are small multiples of 2^-7, so the
elimination is exact; 1e-10 is asked."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(16, 1), (32, 40), (32, 41), (33, 27), (33, 28), (40, 24), (40, 25), (85, 1), (86, 1), (86, 2), (87, 1), (95, 1),
         (95, 2), (96, 1), (97, 1), (112, 17), (257, 2), (300, 3), (700, 1), (1001, 1), (1200, 1), (1201, 1),
         (50, 768), (50, 769), (200, 768)]


@pytest.mark.parametrize("n,nrhs", SIZES)
def test_residual(mh, gpu, n, nrhs):
    rng = np.random.default_rng(n + nrhs)
    A = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    A[np.arange(n), np.arange(n)] *= 1e-3
    b = rng.standard_normal((n, nrhs)) + 1j * rng.standard_normal((n, nrhs))
    X = np.asarray(mh.solve(A, np.eye(n, dtype=complex), b, ctx=gpu)).reshape(n, nrhs)
    res = np.abs(A @ X - b).max(axis=0)
    assert np.all(res <= 8 * n * 2.0 ** -53 * np.abs(A).max() * np.abs(X).max(axis=0))


def _permuted(n, rng):
    U = np.triu(rng.integers(-2, 3, (n, n)).astype(complex), 1) * 2.0 ** -7 + np.eye(n)
    return U, (lambda M: np.roll(M, 29 % n, axis=0))


@pytest.mark.parametrize("n,nrhs", SIZES)
def test_exchanges_at_every_column(mh, gpu, n, nrhs):
    rng = np.random.default_rng(n)
    U, perm = _permuted(n, rng)
    A = perm(U)
    x = rng.integers(-4, 5, (n, nrhs)) + 1j * rng.integers(-4, 5, (n, nrhs))
    X = np.asarray(mh.solve(A, np.eye(n, dtype=complex), A @ x, ctx=gpu)).reshape(n, nrhs)
    assert np.abs(X - x).max() <= 1e-10


@pytest.mark.parametrize("n", [50, 90, 97, 300, 1001, 1200])
@pytest.mark.parametrize("where", ["first", "middle", "last"])
def test_zero_pivot_is_reported(mh, gpu, n, where):
    c = {"first": 0, "middle": n // 2, "last": n - 1}[where]
    U, perm = _permuted(n, np.random.default_rng(n))
    U[c, c] = 0.0
    with pytest.raises(mh.SingularMatrixError, match=f"column {c + 1}$"):
        mh.solve(perm(U), np.eye(n, dtype=complex), np.ones(n, dtype=complex), ctx=gpu)
