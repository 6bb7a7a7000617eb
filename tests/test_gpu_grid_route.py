"""1-D grids below 2^30 pairs under AUTO: the tcgen05 kernel only where it is the faster
one.  A grid of few whole row tiles (128 rows) is the popc kernel's best shape and the
tcgen05 kernel's worst (an operand per column tile, used by a few row tiles); many row
tiles, or a ragged last one, turn that round.  Same bins on either."""
import pytest

import coding_reliability_b200 as dd

pytestmark = pytest.mark.gpu


def grid(A, k, m, kernel):
    return dd.Request(dd.CODE_AN, dd.MODE_GRID_1D, A, k, m=m, kernel=kernel)


def best(call, n=8):
    call()
    return min((call() for _ in range(n)), key=lambda r: r.kernel_ms)


@pytest.mark.parametrize("A,k,m,mma", [(62307, 20, 128, False), (62307, 19, 256, False), (62307, 18, 512, False), (62307, 17, 1024, False),
                                       (62307, 20, 256, False), (62307, 15, 4096, False), (1733, 14, 8192, False), (62307, 17, 4096, True),
                                       (62307, 16, 8192, True), (62307, 16, 2805, True), (62307, 20, 1024, True),
                                       # the popc kernel starts anew every 2^32 / A columns
                                       (2147483659, 16, 2048, True), (2147483659, 20, 256, True), (1073741827, 17, 1024, True),
                                       (16777259, 20, 256, False)])
def test_route(ctx, A, k, m, mma):
    ctx.autotune()
    auto, popc = (best(lambda kern=kern: ctx.histogram(grid(A, k, m, kern))) for kern in (dd.KERNEL_AUTO, dd.KERNEL_POPC))
    assert auto.kernel_used == (dd.KERNEL_MMA if mma else dd.KERNEL_POPC)
    assert auto.raw == popc.raw and auto.counts == popc.counts
    # either the same kernel or a faster one: 15 % for the spread of launches of 40 us and more
    assert auto.kernel_ms <= 1.15 * popc.kernel_ms


@pytest.mark.parametrize("k,m,count,mma", [(18, 256, 16, False), (20, 128, 16, False), (14, 4096, 32, True), (16, 2048, 16, True)])
def test_route_of_a_batch(ctx, k, m, count, mma):
    ctx.autotune()
    As = [32769 + 2 * 997 * i for i in range(count)]
    auto, popc = (best(lambda kern=kern: ctx.batch([grid(A, k, m, kern) for A in As])[0]) for kern in (dd.KERNEL_AUTO, dd.KERNEL_POPC))
    assert auto.kernel_used == (dd.KERNEL_MMA if mma else dd.KERNEL_POPC) and auto.raw == popc.raw
    assert auto.kernel_ms <= 1.15 * popc.kernel_ms
