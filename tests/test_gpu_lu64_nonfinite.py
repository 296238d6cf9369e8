"""Matrices with entries that are no finite numbers in the FP64 solve, as the pivoted
LU of a library treats them: infinite entries end in a column without a number and
are refused as singular (unless only the last pivot is infinite), a NaN is accepted;
its solution is NaN here."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(2, 1), (5, 1), (40, 2), (40, 30), (120, 1), (300, 3)]


def _system(n, nrhs):
    rng = np.random.default_rng(n)
    return (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)),
            rng.standard_normal((n, nrhs)) + 1j * rng.standard_normal((n, nrhs)))


@pytest.mark.parametrize("n,nrhs", SIZES)
def test_infinite_first_column_is_refused(mh, gpu, n, nrhs):
    A, b = _system(n, nrhs)
    for row in (0, n // 2, n - 1):
        M = A.copy()
        M[row, 0] = np.inf
        with pytest.raises(mh.SingularMatrixError, match="column 2$"):
            mh.solve(M, np.eye(n, dtype=complex), b, ctx=gpu)


@pytest.mark.parametrize("n,nrhs", SIZES[1:])
def test_infinite_middle_column_is_refused(mh, gpu, n, nrhs):
    A, b = _system(n, nrhs)
    A[0, n // 2] = np.inf
    with pytest.raises(mh.SingularMatrixError):
        mh.solve(A, np.eye(n, dtype=complex), b, ctx=gpu)


@pytest.mark.parametrize("n,nrhs", SIZES)
@pytest.mark.parametrize("value", [np.nan, complex(0.0, np.nan), complex(np.nan, np.inf)])
def test_nan_is_accepted(mh, gpu, n, nrhs, value):
    A, b = _system(n, nrhs)
    for at in ((0, 0), (n - 1, n - 1), (0, n - 1), (n // 2, 0)):
        M = A.copy()
        M[at] = value
        assert np.isnan(np.asarray(mh.solve(M, np.eye(n, dtype=complex), b, ctx=gpu))).all()


@pytest.mark.parametrize("nrhs", [1, 45])
def test_one_by_one(mh, gpu, nrhs):
    with pytest.raises(mh.SingularMatrixError, match="column 1$"):
        mh.solve(np.array([[np.nan + 0j]]), np.eye(1, dtype=complex), np.ones((1, nrhs), dtype=complex), ctx=gpu)
