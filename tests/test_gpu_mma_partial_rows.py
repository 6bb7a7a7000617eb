"""Grids whose last row tile is not full on the tcgen05 kernel (paired epilogue: a lane's row
counts wholly or not at all in a half tile): rows left over around the warps' 32, windows of every
distance and of a part (outliers included), ragged last columns beside them; against the
popc kernel.  And the time of a grid with such a tile against one without."""
import pytest

import coding_reliability_b200 as dd

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def paired(ctx):
    ctx.set_mma_epilogue(dd.MMA_EPILOGUE_PAIRED)
    yield
    ctx.set_mma_epilogue(dd.MMA_EPILOGUE_AUTO)


def one(A, k, m, kernel):
    return dd.Request(dd.CODE_AN, dd.MODE_GRID_1D, A, k, m=m, kernel=kernel)


def same(ctx, q):
    mma = ctx.histogram(q(dd.KERNEL_MMA))
    popc = ctx.histogram(q(dd.KERNEL_POPC))
    assert (mma.kernel_used, popc.kernel_used) == (dd.KERNEL_MMA, dd.KERNEL_POPC)
    assert mma.raw == popc.raw and mma.counts == popc.counts


@pytest.mark.parametrize("A,k", [(641, 14), (62307, 18), (65537, 22)])
@pytest.mark.parametrize("rest", [1, 31, 32, 33, 64, 96, 104, 127])
def test_rows_left_over(ctx, A, k, rest):
    for rows in (rest, 128 + rest):
        if rows >= 3:
            same(ctx, lambda kern: one(A, k, rows, kern))


@pytest.mark.parametrize("A,k,m,m2", [(61, 44, 1024, 129), (61, 44, 4096, 5001), (58659, 40, 2048, 1000), (58659, 40, 2047, 1000),
                                      (58659, 40, 1025, 33), (145, 46, 3000, 95), (641, 12, 1000, 1000)])
def test_ragged_rows_and_columns(ctx, A, k, m, m2):
    same(ctx, lambda kern: dd.Request(dd.CODE_AN, dd.MODE_GRID_2D, A, k, m=m, m2=m2, kernel=kern))


def test_time_of_a_part_tile(ctx):
    def best(m, n=8):
        q = one(65537, 22, m, dd.KERNEL_MMA)
        ctx.histogram(q)
        return min(ctx.histogram(q).kernel_ms for _ in range(n))

    # three of a tile's four warps' rows, of eight tiles: 1.14 of the time of eight full ones
    # (1.38 through the checked loop, 1.22 before that loop had votes)
    assert best(992) <= 1.2 * best(1024)
