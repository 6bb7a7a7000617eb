"""Popc launches whose tiles have few columns (2-D grids of 17 to 300 columns and many rows):
columns around the parts' edges, against the tcgen05 kernel; and the time of a grid that no
split can shorten, against one that a split halves."""
import pytest

import coding_reliability_b200 as dd

pytestmark = pytest.mark.gpu


def grid(m, m2, kernel=dd.KERNEL_POPC):
    return dd.Request(dd.CODE_AN, dd.MODE_GRID_2D, 58659, 40, m=m, m2=m2, kernel=kernel)


@pytest.mark.parametrize("m", [1, 17, 31, 32, 33, 43, 63, 64, 65, 127, 129, 257, 300])
@pytest.mark.parametrize("m2", [1, 1000, 50000])
def test_few_columns(ctx, m, m2):
    popc, mma = ctx.histogram(grid(m, m2)), ctx.histogram(grid(m, m2, dd.KERNEL_MMA))
    assert (popc.kernel_used, mma.kernel_used) == (dd.KERNEL_POPC, dd.KERNEL_MMA)
    assert popc.raw == mma.raw and popc.counts == mma.counts


@pytest.mark.parametrize("k,m", [(9, 1), (12, 64), (12, 85), (12, 86), (13, 128), (13, 255)])
def test_few_codewords_a_lane(ctx, k, m):
    """Monte Carlo tiles of one to 64 codewords a lane: parts are whole codewords."""
    import oracle
    q = dd.Request(dd.CODE_AN, dd.MODE_MONTE_CARLO, 58659, k, m=m, seed=11)
    nb, h, A = dd.request_shape(q)
    assert ctx.histogram(q).raw == oracle.an_mc_raw(A, k, m, q.seed, nb)


def test_empty_parts_are_not_claimed(ctx):
    def best(m, m2, n=30):
        ctx.histogram(grid(m, m2))
        return min(ctx.histogram(grid(m, m2)).kernel_ms for _ in range(n))

    # 17 of a tile's 1024 columns, 782 row tiles (16.9 us) against eight (14.6): with each of
    # the former claimed in 16 parts 23 us
    assert best(17, 100000) <= 1.35 * best(17, 1000)
