"""Packed fields of the folding kernel (dd_carry.cu, windows of 5 and 6 bits): multipliers
2^j + 1, whose windows fill the 16-bit fields furthest (two thirds with six window bits, by
a model of the kernel's columns and rows), and 2^j - 1.  No instance may be counted
again by a pair kernel, alone or in a batch, whose rows are cut into other segments."""
import pytest

import coding_reliability_b200 as dd

pytestmark = pytest.mark.gpu

CASES = [(33, 12), (65, 13), (129, 14), (257, 15), (513, 16), (1025, 17), (2049, 18), (4097, 19), (8193, 20), (16385, 21), (32769, 22),
         (33, 11), (513, 15), (4097, 18), (16385, 20), (511, 15), (1023, 16), (8191, 19)]


def req(A, k, kernel):
    return dd.Request(dd.CODE_AN, dd.MODE_EXHAUSTIVE, A, k, kernel=kernel)


@pytest.mark.parametrize("A,k", CASES)
def test_fullest_fields(ctx, A, k):
    mma = ctx.histogram(req(A, k, dd.KERNEL_MMA))
    for _ in range(3):
        res = ctx.histogram(req(A, k, dd.KERNEL_CARRY))
        assert res.kernel_used == dd.KERNEL_CARRY
        assert res.raw == mma.raw and res.counts == mma.counts


def test_fullest_fields_batch(ctx):
    qs = [req(A, k, dd.KERNEL_CARRY) for A, k in CASES if k <= 20]
    want = [ctx.histogram(req(q.A, q.n, dd.KERNEL_MMA)).raw for q in qs]
    for graph in (False, True, True):
        out = ctx.batch(qs, use_graph=graph)
        assert [r.kernel_used for r in out] == [dd.KERNEL_CARRY] * len(qs)
        assert [r.raw for r in out] == want
