"""The residue-pair kernels (dd_carry.cu) against the oracle and the tcgen05
kernel, bit-exact: every window length (k - bits(A) = 1..8 levels, one kernel up to
4, staged above), residues hit by one, two and many q, and residue counts at the
edges of the column strips (112 and 177 useful columns), row segments and staged
blocks (about 3580 residues a side).  The 1-D grid form (dd_carry_rows.cu): rows
in blocks of a power-of-two stride and listed rows, strips of 449 and 769 useful
columns, few and many columns a residue, several slices of them, and all residues in
one CTA (A <= 512 and <= 1024)."""
import pytest

import coding_reliability_b200 as dd
import oracle

pytestmark = pytest.mark.gpu


def req(A, k, kernel, **kw):
    return dd.Request(dd.CODE_AN, dd.MODE_EXHAUSTIVE, A, k, kernel=kernel, **kw)


@pytest.mark.parametrize("A,k", [(1, 2), (1, 9), (3, 3), (3, 12), (5, 4), (7, 13), (33, 7), (61, 8), (61, 13), (63, 10),
                                 (91, 13), (113, 12), (115, 11), (225, 12), (243, 12), (255, 9), (257, 13), (353, 11), (511, 13)])
def test_carry_vs_oracle(ctx, A, k):
    q = req(A, k, dd.KERNEL_CARRY)
    nb, h, Aeff = dd.request_shape(q)
    res = ctx.histogram(q)
    assert res.kernel_used == dd.KERNEL_CARRY
    assert res.raw == oracle.an_exhaustive_raw(Aeff, k, nb)
    assert res.counts == oracle.an_exhaustive_counts(Aeff, k, nb)


@pytest.mark.parametrize("A,k", [(4097, 14), (4819, 15), (4033, 16), (8191, 17), (32769, 17), (65535, 18),  # one kernel
                                 (33, 14), (867, 20), (129, 16),                       # staged, many q per residue
                                 (3583, 17), (3585, 18), (3577, 19), (3579, 19), (3569, 20), (3571, 21), (4097, 19), (7163, 18), (12161, 19), (40001, 21)])
def test_carry_vs_tcgen05(ctx, A, k):
    res = ctx.histogram(req(A, k, dd.KERNEL_CARRY))
    mma = ctx.histogram(req(A, k, dd.KERNEL_MMA))
    assert (res.kernel_used, mma.kernel_used) == (dd.KERNEL_CARRY, dd.KERNEL_MMA)
    assert res.raw == mma.raw and res.counts == mma.counts and res.minb == mma.minb


@pytest.mark.parametrize("A,k", [(9, 14), (11, 12), (11, 17), (13, 14), (17, 13), (23, 12), (31, 16), (61, 19), (129, 18),
                                 (301, 13), (581, 20), (867, 14), (723, 15)])
def test_carry_short_segments(ctx, A, k):
    """Segments of 4 and 8 rows: shorter than the rows a segment computes twice."""
    res = ctx.histogram(req(A, k, dd.KERNEL_CARRY))
    popc = ctx.histogram(req(A, k, dd.KERNEL_POPC))
    assert (res.kernel_used, popc.kernel_used) == (dd.KERNEL_CARRY, dd.KERNEL_POPC)
    assert res.raw == popc.raw and res.counts == popc.counts


@pytest.mark.parametrize("A,k", [(33, 11), (33, 12), (63, 11), (63, 12), (129, 13), (255, 14), (4095, 17), (4095, 18), (3583, 18),
                                 (16385, 20), (32767, 21), (32769, 21), (65535, 21), (58659, 21), (65521, 22)])
def test_carry_packed_fold(ctx, A, k):
    """Windows of 5 and 6 bits: one and two folded levels, one and two q per residue,
    16-bit q (whose last neighbour is past the table's distances)."""
    res = ctx.histogram(req(A, k, dd.KERNEL_CARRY))
    mma = ctx.histogram(req(A, k, dd.KERNEL_MMA))
    assert (res.kernel_used, mma.kernel_used) == (dd.KERNEL_CARRY, dd.KERNEL_MMA)
    assert res.raw == mma.raw and res.counts == mma.counts


@pytest.mark.parametrize("A,k", [(3, 14), (3, 18), (5, 20), (31, 15), (33, 15), (63, 20), (65, 16), (255, 18), (511, 19), (1019, 21),
                                 (1023, 20), (2047, 21), (8191, 23)])
def test_carry_many_q(ctx, A, k):
    """Many q per residue: sums in registers, and the wide products of the shortest A."""
    res = ctx.histogram(req(A, k, dd.KERNEL_CARRY))
    mma = ctx.histogram(req(A, k, dd.KERNEL_MMA))
    assert (res.kernel_used, mma.kernel_used) == (dd.KERNEL_CARRY, dd.KERNEL_MMA)
    assert res.raw == mma.raw and res.counts == mma.counts


def test_carry_batch(ctx):
    """Jobs of one launch: more than a launch's 32 entries, every window length, few
    and many q, and staged blocks that need several rounds."""
    qs = [req(A, k, dd.KERNEL_CARRY) for k in (12, 13) for A in range(33, 33 + 2 * 40, 2)]
    qs += [req(A, 14, dd.KERNEL_CARRY) for A in (1, 5, 17, 63, 255, 511, 1023, 2047, 4095, 8191)]
    qs += [req(A, 17, dd.KERNEL_CARRY) for A in (4001, 4003, 4005, 4007)]
    want = [ctx.histogram(req(q.A, q.n, dd.KERNEL_POPC)).raw for q in qs]
    for graph in (False, True, True):
        out = ctx.batch(qs, use_graph=graph, kernel=dd.KERNEL_CARRY)
        for q, r, w in zip(qs, out, want):
            assert r.kernel_used == dd.KERNEL_CARRY and r.raw == w, (q.A, q.n)


def grid(A, k, m, kernel, **kw):
    return dd.Request(dd.CODE_AN, dd.MODE_GRID_1D, A, k, m=m, kernel=kernel, **kw)


@pytest.mark.parametrize("A,k,m", [(1, 12, 64), (3, 12, 13), (5, 13, 4096), (61, 12, 4096), (449, 12, 65), (451, 13, 64),
                                   (641, 14, 1000), (1023, 13, 3), (771, 12, 17), (1021, 15, 333), (976, 14, 128),
                                   (1, 13, 100), (33, 14, 777), (511, 13, 2047), (513, 12, 1001), (1537, 13, 99)])
def test_grid_vs_oracle(ctx, A, k, m):
    q = grid(A, k, m, dd.KERNEL_CARRY)
    nb, h, Aeff = dd.request_shape(q)
    res = ctx.histogram(q)
    assert res.kernel_used == dd.KERNEL_CARRY
    assert res.raw == oracle.an_grid1d_raw(Aeff, k, h, m, nb)[0]


@pytest.mark.parametrize("A,k,m", [(65535, 16, 256), (65535, 20, 100), (32769, 24, 128), (8191, 22, 1 << 12),
                                   (1283, 24, 99), (61, 24, 1 << 10), (33, 27, 64), (35, 25, 21), (65535, 27, 64), (127, 24, 301),
                                   (33, 23, 1001), (867, 22, 333), (1027, 22, 333)])
def test_grid_vs_tcgen05(ctx, A, k, m):
    res = ctx.histogram(grid(A, k, m, dd.KERNEL_CARRY))
    mma = ctx.histogram(grid(A, k, m, dd.KERNEL_MMA))
    assert (res.kernel_used, mma.kernel_used) == (dd.KERNEL_CARRY, dd.KERNEL_MMA)
    assert res.raw == mma.raw and res.counts == mma.counts and res.minb == mma.minb


def test_route(ctx):
    """AUTO takes the path where its rule says so, for a batch's jobs one by one; an
    even multiplier (kept by the CPU convention) counts as its odd part; jobs outside
    the path's range run on a pair kernel although it is asked for."""
    qs = [req(641, 14, dd.KERNEL_AUTO), req(641, 13, dd.KERNEL_AUTO), req(1283, 14, dd.KERNEL_AUTO),
          req(976, 15, dd.KERNEL_AUTO, convention=dd.CONV_CPU), req(61, 15, dd.KERNEL_POPC),
          req(131071, 12, dd.KERNEL_CARRY), req(641, 10, dd.KERNEL_CARRY),
          grid(641, 18, 1024, dd.KERNEL_AUTO), grid(641, 18, 1023, dd.KERNEL_AUTO), grid(641, 18, 1025, dd.KERNEL_AUTO),
          grid(641, 11, 64, dd.KERNEL_CARRY)]
    want = [True, False, False, True, False, False, False, True, False, True, False]  # which pair kernel is the autotuner's
    for graph in (False, True, True):
        out = ctx.batch(qs, use_graph=graph)
        assert [r.kernel_used == dd.KERNEL_CARRY for r in out] == want
        for q, r in zip(qs, out):
            p = ctx.histogram(dd.Request(q.code, q.mode, q.A, q.n, m=q.m, convention=q.convention, kernel=dd.KERNEL_POPC))
            assert r.raw == p.raw and r.counts == p.counts and r.pairs == p.pairs


@pytest.mark.parametrize("A,k,carry", [(32769, 19, True), (45875, 19, True), (45877, 19, False), (65535, 19, False), (22937, 18, True),
                                       (22939, 18, False), (2 * 22937, 18, True), (8193, 17, False), (32769, 18, False)])
def test_route_three_bits(ctx, A, k, carry):
    """k three bits above A's: the residues of the shorter multipliers, codewords for the others."""
    ctx.autotune()
    res = ctx.histogram(req(A, k, dd.KERNEL_AUTO))
    assert res.kernel_used == (dd.KERNEL_CARRY if carry else dd.KERNEL_MMA)
    other = ctx.histogram(req(A, k, dd.KERNEL_MMA if carry else dd.KERNEL_CARRY))
    assert res.raw == other.raw and res.counts == other.counts
