"""Launches of few tiles on the popc kernel, whose warps claim parts of a tile: sizes
around the parts' edges (32 columns, 128 rows), Monte Carlo blocks cut short at either
end, sampled Ext-Hamming weights with a ragged last block; against the oracle."""
import pytest

import coding_reliability_b200 as dd
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("A,k", [(3, 1), (641, 6), (641, 7), (58659, 8), (65535, 10), (1021, 11), (65521, 17)])
def test_exhaustive_parts(ctx, A, k):
    q = dd.Request(dd.CODE_AN, dd.MODE_EXHAUSTIVE, A, k, kernel=dd.KERNEL_POPC)
    nb, h, Aeff = dd.request_shape(q)
    res = ctx.histogram(q)
    assert res.kernel_used == dd.KERNEL_POPC and res.raw == oracle.an_exhaustive_raw(Aeff, k, nb)


@pytest.mark.parametrize("A,k,m,seed", [(61, 5, 3, 1), (641, 8, 15, 2), (641, 8, 256, 3), (58659, 9, 255, 4),
                                        (58659, 10, 257, 5), (65535, 11, 1031, 6), (58659, 18, 5, 7)])
def test_monte_carlo_parts(ctx, A, k, m, seed):
    q = dd.Request(dd.CODE_AN, dd.MODE_MONTE_CARLO, A, k, m=m, seed=seed << 33 | 5)
    nb, h, Aeff = dd.request_shape(q)
    res = ctx.histogram(q)
    m = min(m, 1 << k)
    assert res.raw == oracle.an_mc_raw(Aeff, k, m, q.seed, nb)
    done = m // 2  # a continued run starts inside a block
    if done:
        first = ctx.histogram(dd.Request(dd.CODE_AN, dd.MODE_MONTE_CARLO, A, k, m=done, seed=q.seed))
        assert ctx.mc_extend(q, done, first.raw).raw == res.raw


@pytest.mark.parametrize("n,m", [(8, 7), (8, 256), (16, 33), (16, 8191), (24, 8193), (32, 100003), (40, 100003), (48, 70000)])
def test_hamming_parts(ctx, n, m):
    for mode in (dd.MODE_MONTE_CARLO, dd.MODE_GRID_1D):
        q = dd.Request(dd.CODE_EXT_HAMMING, mode, 1, n, m=m, seed=99, with_1bit=1)
        nb, h, _ = dd.request_shape(q)
        res = ctx.histogram(q)
        raw, _ = oracle.hamming_mc_raw(n, m, 99, nb) if mode == dd.MODE_MONTE_CARLO else oracle.hamming_grid_raw(n, m, nb)
        assert res.raw == raw
