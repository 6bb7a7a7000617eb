"""1-D grids of the shortest multipliers under AUTO: the residue route only where it is the
faster one, k on both sides of the cyclic form's (24), listed rows and rows in blocks."""
import pytest

import coding_reliability_b200 as dd

pytestmark = pytest.mark.gpu


def grid(A, k, m, kernel):
    return dd.Request(dd.CODE_AN, dd.MODE_GRID_1D, A, k, m=m, kernel=kernel)


@pytest.mark.parametrize("A,k,m,carry", [(1, 25, 1000, False), (3, 25, 1000, False), (3, 26, 384, False), (1, 25, 129, False), (1, 25, 100, False),
                                         (3, 25, 300, True), (5, 25, 1000, False), (1, 25, 50, True), (5, 25, 500, True), (7, 25, 1000, True),
                                         (1, 24, 1000, True), (1, 18, 1024, False), (3, 20, 256, False),
                                         (5, 20, 256, False), (13, 21, 128, False), (15, 21, 128, True), (1, 22, 64, True), (1, 20, 1024, True)])
def test_route(ctx, A, k, m, carry):
    ctx.autotune()

    def best(kernel, n=6):
        ctx.histogram(grid(A, k, m, kernel))
        return min((ctx.histogram(grid(A, k, m, kernel)) for _ in range(n)), key=lambda r: r.kernel_ms)

    auto = best(dd.KERNEL_AUTO)
    assert (auto.kernel_used == dd.KERNEL_CARRY) == carry
    others = [best(kern) for kern in (dd.KERNEL_POPC, dd.KERNEL_MMA, dd.KERNEL_CARRY)]
    assert all(r.raw == auto.raw and r.counts == auto.counts for r in others)
    # the faster of the two that a program could have had before the residue route
    assert auto.kernel_ms <= 1.1 * (others[0] if (m << k) < 1 << 30 else others[1]).kernel_ms
