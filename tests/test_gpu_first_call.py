"""The first calls of a context: the autotuner (a second of probes) runs before the first
launch whose kernel depends on its verdict, not before residue-route calls that asked for it;
later calls get the verdict as if it had run at once."""
import time

import pytest

import coding_reliability_b200 as dd

pytestmark = pytest.mark.gpu

# the autotuner's twelve runs of k = 20 take 1.2 s; a residue call with its first
# allocations a few ms
LIMIT_S = 0.4


def an(A, k, **kw):
    return dd.Request(dd.CODE_AN, dd.MODE_EXHAUSTIVE, A, k, **kw)


def seconds(call):
    t = time.perf_counter()
    res = call()
    return time.perf_counter() - t, res


@pytest.fixture
def fresh(ctx):
    # kernel images are loaded once a process: by the session's context
    ctx.histogram(an(867, 21))
    ctx.batch([an(129 + 2 * i, 14) for i in range(16)], use_graph=True)
    c = dd.Context(0)
    yield c
    c.close()


def test_residue_call_is_not_tuned_for(fresh):
    t, res = seconds(lambda: fresh.histogram(an(867, 21)))
    assert res.kernel_used == dd.KERNEL_CARRY and t < LIMIT_S
    # the verdict it asked for is there when a call reads it, whose own time leaves the probes out
    t, res = seconds(lambda: fresh.histogram(an(58659, 16)))
    assert res.kernel_used == dd.KERNEL_MMA and t > LIMIT_S and res.total_ms < 1e3 * LIMIT_S
    t, res = seconds(lambda: fresh.histogram(an(58659, 16)))
    assert res.kernel_used == dd.KERNEL_MMA and t < LIMIT_S


def test_residue_batch_is_not_tuned_for(fresh):
    t, out = seconds(lambda: fresh.batch([an(129 + 2 * i, 14) for i in range(16)], use_graph=True))
    assert all(r.kernel_used == dd.KERNEL_CARRY for r in out) and t < LIMIT_S
    t, out = seconds(lambda: fresh.batch([an(58659, 8)] * 16, use_graph=True))
    assert all(r.kernel_used == dd.KERNEL_POPC for r in out) and t < LIMIT_S
    q = dd.Request(dd.CODE_AN, dd.MODE_GRID_2D, 641, 40, m=20000, m2=20000)
    assert fresh.histogram(q).kernel_used == dd.KERNEL_MMA


def test_pair_kernel_call_is_tuned_for(fresh):
    res = fresh.histogram(an(62307, 20, kernel=dd.KERNEL_POPC))  # names its kernel: no probe
    assert res.kernel_used == dd.KERNEL_POPC
    assert fresh.histogram(an(58659, 16)).kernel_used == dd.KERNEL_POPC  # nothing asked for one yet
    res = fresh.histogram(an(65537, 20))  # 17 bits: no residue route
    assert res.kernel_used == dd.KERNEL_MMA
    assert fresh.histogram(an(58659, 16)).kernel_used == dd.KERNEL_MMA


def test_part_after_residue_call(fresh):
    """A part of a request runs on the kernel the verdict gives, and adds up as before."""
    fresh.histogram(an(867, 21))
    q = an(58659, 16)
    tiles = dd.request_plan(q)["tiles"]
    raw = None
    for lo, n in ((0, 100), (100, tiles - 100)):
        raw, _ = fresh.histogram_part(q, lo, n, raw)
    res = fresh.histogram(q)
    assert raw == res.raw
