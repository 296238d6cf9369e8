"""The tensor-core LU of few matrices: the next diagonal block is updated by a
kernel of its own (64 x 64) and the rest of its tile by the strip, so the sizes
go through blocks at the start and in the middle of a 128-wide tile, ragged last
blocks and tiles, odd orders (no bulk copies) and steps with several panels
deferred.

Tolerance: the products are of FP16 operands (unit roundoff u = 2^-11) summed in
FP32, so A - LU has entries of about u |L||U|; the matrices are diagonally
dominant with |L||U| <= 2 |A| + small, rows summed over sqrt(n) random terms.
8 u = 3.9e-3 of max |A| covers them (a missed or doubled 64-column update is of
the size of the off-diagonal entries' products, 1 / n of the diagonal, times n)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _matrices(nb, n, seed):
    rng = np.random.default_rng(seed)
    A = rng.standard_normal((nb, n, n)) + 1j * rng.standard_normal((nb, n, n))
    return A / np.sqrt(2.0 * n) + 2.0 * np.eye(n)


@pytest.mark.parametrize("schedule", [(1, 2, 0), (1, 4, 0), (1, 4, 1), (1, 8, 0)])
@pytest.mark.parametrize("n", [64, 65, 128, 129, 192, 193, 256, 320, 383, 448, 700])
def test_block_update(gpu, n, schedule):
    keep = gpu.lu_schedule(n)
    try:
        gpu.set_lu_schedule(n, *schedule)
        A = _matrices(2, n, n)
        F, bad = gpu.lu_factor_lowp(A, backend="tcgen05")
    finally:
        gpu.set_lu_schedule(n, *keep)
    assert not np.any(bad)
    F = np.asarray(F, dtype=np.complex128)
    for a, f in zip(A, F):
        L = np.tril(f, -1) + np.eye(n)
        U = np.triu(f)
        assert np.abs(L @ U - a).max() <= 8 * 2.0 ** -11 * np.abs(a).max()
