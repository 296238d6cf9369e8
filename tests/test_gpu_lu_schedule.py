"""Which schedule a factorisation runs: the built-in entries by the size and the
call's columns in all, and that saving and restoring a size's entry, or setting
its built-in values, leaves every size as a new context has it."""
import pytest

pytestmark = pytest.mark.gpu

SIZES = (64, 512, 600, 724, 725, 777, 846, 1024, 1253, 1254, 1640, 1773, 1774, 2048, 4096)


@pytest.fixture
def ctx(mh, gpu):
    c = mh.Context(0)
    yield c
    c.close()


def _runs(ctx):
    return {(n, nb): ctx.lu_schedule(n, nb) for n in SIZES for nb in (1, 16, 17, 31, 32, 33, 64)}


def test_entries_by_columns(ctx):
    for n, at, above in ((2048, (1, 4, 0), (2, 8, 0)), (1024, (1, 4, 0), (2, 4, 0)), (1536, (1, 4, 0), (2, 4, 0)),
                         (512, (1, 4, 1), (1, 4, 1))):
        most = 32768 // n
        assert ctx.lu_schedule(n, 1) == ctx.lu_schedule(n, most) == at
        assert ctx.lu_schedule(n, most + 1) == ctx.lu_schedule(n, 1000) == above


def test_restoring_leaves_a_new_table(ctx):
    new = _runs(ctx)
    for n in SIZES:
        keep = ctx.lu_schedule(n)
        other = (3, 6, 1) if keep != (3, 6, 1) else (2, 2, 0)
        ctx.set_lu_schedule(n, *other)
        assert ctx.lu_schedule(n) == ctx.lu_schedule(n, 1) == ctx.lu_schedule(n, 64) == other
        ctx.set_lu_schedule(n, *keep)
    assert _runs(ctx) == new


def test_a_set_entry_stays_and_serves_its_neighbours(ctx):
    ctx.set_lu_schedule(1000, 1, 4, 0)   # what 1000 has: for 1000 alone
    ctx.set_lu_schedule(1024, 3, 2, 0)
    assert ctx.lu_schedule(1000, 1) == (1, 4, 0) and ctx.lu_schedule(1000, 64) == (2, 4, 0)
    assert ctx.lu_schedule(990, 1) == ctx.lu_schedule(990, 64) == (3, 2, 0)


def test_tuned_entry_runs_as_it_was_timed(ctx):
    out = ctx.autotune_lu(256, 2, [(1, 4, 1)])   # the values of the entry 256 has
    assert out["best"] == (1, 4, 1)
    out = ctx.autotune_lu(1024, 1, [(1, 4, 0)])  # the built-in values, without their rule
    assert ctx.lu_schedule(1024, 64) == out["best"] == (1, 4, 0)
