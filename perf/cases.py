"""Performance cases of the distance-distribution library: the calls its users
make, over the range of sizes they make them at, through the public Python API.

A case names the code, the mode, the data bits k, the bit width of the AN
multiplier A and the sample counts; the multipliers themselves (and the Monte
Carlo keys) come from the seed.  A program of this kind keeps one context for
its life and lets it autotune once, so every case uses the same context.
Outputs are whole histograms (the raw device bins and the 128-bit counts as two
64-bit halves) with the minimum distance and its count: whole numbers only.
"""
from __future__ import annotations

import random

import numpy as np

import coding_reliability_b200 as dd

_ctx = None


def _context() -> dd.Context:
    global _ctx
    if _ctx is None:
        _ctx = dd.Context(0)
        _ctx.autotune()
    return _ctx


def listed() -> list[dict]:
    return [
        # one small code: a launch, two copies and the host work around them
        {"name": "exhaustive_k8", "kind": "exhaustive", "k": 8, "a_bits": 8},
        # one 16-bit super-A candidate at the width the sweeps run at
        {"name": "exhaustive_k16", "kind": "exhaustive", "k": 16, "a_bits": 16},
        # one candidate at the widest data the serving mix asks for exhaustively
        {"name": "exhaustive_k20", "kind": "exhaustive", "k": 20, "a_bits": 16},
        # a short multiplier (the published tables use 6 to 10 bits) over wide data
        {"name": "exhaustive_k21_a10", "kind": "exhaustive", "k": 21, "a_bits": 10},
        # the largest exhaustive call: 40-bit-class codewords, one instance
        {"name": "exhaustive_k22", "kind": "exhaustive", "k": 22, "a_bits": 16},
        # super-A sweep: 256 candidates of one width in one batched call
        {"name": "batch_k16", "kind": "batch", "k": 16, "a_bits": 16, "count": 256},
        # super-A search over short multipliers of every width, an odd count
        {"name": "batch_k12_mixed", "kind": "batch", "k": 12, "a_bits": 0, "count": 63},
        # 1-D grid with a power-of-two stride, as the serving mix asks for it
        {"name": "grid1d_k24", "kind": "grid1d", "k": 24, "a_bits": 16, "m": 65536},
        # 1-D grid with a ragged stride, as the grid-convergence studies run it
        {"name": "grid1d_k24_ragged", "kind": "grid1d", "k": 24, "a_bits": 10, "m": 10001},
        # 2-D grid of a code too wide for any exhaustive run
        {"name": "grid2d_k40", "kind": "grid2d", "k": 40, "a_bits": 8, "m": 100001, "m2": 33333},
        # Monte Carlo estimate of a 40-bit code, many samples per codeword
        {"name": "mc_k24", "kind": "mc", "k": 24, "a_bits": 16, "m": 257},
        # Ext-Hamming weight estimate by Monte Carlo
        {"name": "hamming_mc_n40", "kind": "hamming_mc", "k": 40, "a_bits": 0, "m": 1 << 24},
    ]


def _log_int(rng: random.Random, lo: int, hi: int) -> int:
    """An integer in [lo, hi], spread over its logarithm."""
    import math
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng: random.Random) -> dict:
    kind = rng.choice(["exhaustive", "exhaustive", "exhaustive", "batch", "batch", "grid1d", "grid1d", "grid2d", "mc",
                       "hamming_mc"])
    a = rng.randint(6, 16)
    if kind == "exhaustive":
        return {"kind": kind, "k": rng.randint(8, 22), "a_bits": a, "offset": rng.randrange(1 << 14)}
    if kind == "batch":
        # the whole batch stays below 2^40 pairs
        k = rng.randint(8, 16)
        return {"kind": kind, "k": k, "a_bits": rng.choice([0, a, 16]), "count": _log_int(rng, 3, 256)}
    if kind == "grid1d":
        k = rng.randint(12, 24)
        # below 2^40 pairs; half of the draws use a power-of-two stride
        m = 1 << rng.randint(4, min(k, 16)) if rng.random() < 0.5 else _log_int(rng, 13, min(1 << k, 65536))
        return {"kind": kind, "k": k, "a_bits": a, "m": m}
    if kind == "grid2d":
        k = rng.randint(16, 44)
        hi = min(1 << k, 200000)
        return {"kind": kind, "k": k, "a_bits": a, "m": _log_int(rng, 17, hi), "m2": _log_int(rng, 17, hi)}
    if kind == "mc":
        # at most about 2^33 samples in all, few or many per codeword
        k = rng.randint(10, 32)
        return {"kind": kind, "k": k, "a_bits": a, "m": _log_int(rng, 1, max(1, min(1 << k, 1 << (33 - k), 100001)))}
    return {"kind": kind, "k": rng.choice([16, 24, 32, 40]), "a_bits": 0, "m": _log_int(rng, 4096, 1 << 26)}


def _multiplier(rng: random.Random, a_bits: int) -> int:
    """An odd multiplier of exactly a_bits bits (0: of 6 to 16 bits, drawn)."""
    a = a_bits or rng.randint(6, 16)
    return (1 << (a - 1)) | rng.getrandbits(a - 1) | 1


def _own_multiplier(seed: int, a_bits: int) -> int:
    """The odd multiplier of a single instance: neighbouring seeds give different ones."""
    return (1 << (a_bits - 1)) | (seed * 0x9E3779B1 % (1 << (a_bits - 2))) << 1 | 1


def _requests(case: dict, seed: int) -> list[dd.Request]:
    rng = random.Random(seed)
    kind, k = case["kind"], case["k"]
    A = _own_multiplier(seed + case.get("offset", 0), case["a_bits"]) if case["a_bits"] else 1
    if kind == "exhaustive":
        return [dd.Request(dd.CODE_AN, dd.MODE_EXHAUSTIVE, A, k)]
    if kind == "batch":
        return [dd.Request(dd.CODE_AN, dd.MODE_EXHAUSTIVE, _multiplier(rng, case["a_bits"]), k,
                           convention=dd.CONV_SUPER_A) for _ in range(case["count"])]
    if kind == "grid1d":
        return [dd.Request(dd.CODE_AN, dd.MODE_GRID_1D, A, k, m=case["m"])]
    if kind == "grid2d":
        return [dd.Request(dd.CODE_AN, dd.MODE_GRID_2D, A, k, m=case["m"], m2=case["m2"])]
    if kind == "mc":
        return [dd.Request(dd.CODE_AN, dd.MODE_MONTE_CARLO, A, k, m=case["m"], seed=rng.getrandbits(48))]
    if kind == "hamming_mc":
        return [dd.Request(dd.CODE_EXT_HAMMING, dd.MODE_MONTE_CARLO, 1, k, m=case["m"], seed=rng.getrandbits(48),
                           with_1bit=1)]
    raise ValueError(kind)


def prepare(case: dict, seed: int) -> dict:
    return {"ctx": _context(), "batch": case["kind"] == "batch", "requests": _requests(case, seed)}


def _halves(values: list[int]) -> np.ndarray:
    """uint128 values as (low, high) 64-bit halves."""
    return np.array([[v & 0xFFFFFFFFFFFFFFFF for v in values], [v >> 64 for v in values]], dtype=np.uint64).view(np.int64)


def _outputs(results: list) -> list:
    raw = np.zeros((len(results), dd.MAX_BINS), dtype=np.uint64)
    for i, r in enumerate(results):
        raw[i, :r.nbins] = r.raw
    counts = _halves([c for r in results for c in r.counts + [0] * (dd.MAX_BINS - r.nbins)])
    least = _halves([x for r in results for x in (r.minb, r.mincb)])
    return [raw.view(np.int64), counts, least]


def run(state: dict) -> list:
    ctx, reqs = state["ctx"], state["requests"]
    if state["batch"]:
        return _outputs(ctx.batch(reqs, use_graph=True))
    return _outputs([ctx.histogram(reqs[0])])


def _pairs(case: dict) -> int:
    N = 1 << case["k"]
    if case["kind"] == "exhaustive":
        return N * (N - 1) // 2
    if case["kind"] == "batch":
        return case["count"] * (N * (N - 1) // 2)
    if case["kind"] == "grid1d":
        return N * min(N, case["m"])
    if case["kind"] == "grid2d":
        return min(N, case["m"]) * min(N, case["m2"])
    if case["kind"] == "mc":
        return N * min(N, case["m"])
    return min(N, case["m"])


def work(case: dict) -> dict:
    """One distance counted per pair (or weight per sample); the request read and the result written once."""
    n = case.get("count", 1)
    return {"bytes": n * (80 + 3 * 8 * dd.MAX_BINS), "flops": _pairs(case)}


def exact(case: dict, seed: int):
    """The exhaustive histograms by enumeration in 64-bit integers, where that takes seconds."""
    if case["kind"] not in ("exhaustive", "batch") or _pairs(case) > 1 << 27:
        return None
    k = case["k"]
    x = np.arange(1 << k, dtype=np.uint64)
    raw = np.zeros((case.get("count", 1), dd.MAX_BINS), dtype=np.uint64)
    counts, least = [], []
    for i, q in enumerate(_requests(case, seed)):
        c = x * np.uint64(q.A)
        for j in range(1, 1 << k):
            raw[i] += np.bincount(np.bitwise_count(c[j:] ^ c[:-j]), minlength=dd.MAX_BINS).astype(np.uint64)
        # check bits: ceil(log2 A), or the bit length of A in the super-A convention; A is odd and above 1
        nbins = k + (q.A - 1 if q.convention == dd.CONV_GPU else q.A).bit_length() + 1
        t = [1 << k] + [2 * int(v) for v in raw[i, 1:nbins]]
        lim = (nbins + 1) // 2 if q.convention == dd.CONV_SUPER_A else nbins // 2
        first = next((d for d in range(1, lim) if t[d]), None)
        counts += t + [0] * (dd.MAX_BINS - nbins)
        least += [0xFFFF, (1 << 128) - 1] if first is None else [first, t[first]]
    return [raw.view(np.int64), _halves(counts), _halves(least)]
