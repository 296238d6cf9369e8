"""The tensor-core LU of few matrices entry by entry (the sizes and schedules of
test_gpu_lu_few.py): blocks at the start and in the middle of a 128-wide tile, ragged
last blocks and tiles, odd orders, steps with several panels deferred.

Bound: every product takes operands rounded to FP16 (2^-12 of an entry), so an entry
of A - L U is off by at most about 2^-11 of the same entry of |L| |U|, without the
exact l_ii u_ii, once for the update and once for the panel solve's product with an
inverse block.  The same elimination in numpy with rounded operands reaches 8e-4 of
it; 2^-9 is asked, with 1e-2 of the scale for FP32.  Six entries missed by one
64-column update are 0.1 or more (planted there)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("schedule", [(1, 2, 0), (1, 4, 0), (1, 4, 1), (1, 8, 0), (2, 4, 0)])
@pytest.mark.parametrize("n", [64, 65, 128, 129, 192, 193, 256, 320, 383, 448, 700])
def test_entries(mh, gpu, n, schedule):
    rng = np.random.default_rng(n)
    A = rng.standard_normal((2, n, n)) + 1j * rng.standard_normal((2, n, n))
    A = A / np.sqrt(2.0 * n) + 2.0 * np.eye(n)
    ctx = mh.Context(0)
    try:
        ctx.set_lu_schedule(n, *schedule)
        F, bad = ctx.lu_factor_lowp(A, backend="tcgen05")
    finally:
        ctx.close()
    assert not np.any(bad)
    for a, f in zip(A, np.asarray(F, dtype=np.complex128)):
        L, U = np.tril(f, -1) + np.eye(n), np.triu(f)
        scale = np.abs(L) @ np.abs(U) - np.diag(np.abs(np.diag(U))) + 1e-2
        assert np.all(np.abs(L @ U - a) <= 2.0 ** -9 * scale)
