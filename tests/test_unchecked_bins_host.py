"""The Monte Carlo kernels and the sampled Ext-Hamming weights (dd_kernels.cu) add to bins
without a range check: every distance or weight of a request that the shape rules accept has
to lie below its nbins.  Codewords of n + h bits are distances up to nbins - 1; a sampled
message of the code's N bits has at most N plus its 4, 5 or 6 parity bits set."""
import random

import pytest

import coding_reliability_b200 as dd


def accepted(q):
    try:
        return dd.request_shape(q)
    except dd.DDError:
        return None


@pytest.mark.parametrize("convention", [dd.CONV_GPU, dd.CONV_SUPER_A])
def test_monte_carlo_codewords_fit(lib, convention):
    rng = random.Random(7)
    edges = [v for b in range(33) for v in ((1 << b) - 1, 1 << b, (1 << b) + 1)]
    taken = refused = 0
    for n in range(1, 49):
        for A in edges + [rng.randrange(1 << rng.randint(1, 32)) for _ in range(40)]:
            for h in (0, rng.randint(1, 40), max(1, A.bit_length() - 1)):
                s = accepted(dd.Request(dd.CODE_AN, dd.MODE_MONTE_CARLO, A, n, m=5, h=h, convention=convention))
                if s is None:
                    refused += 1
                    continue
                nbins, _, eff = s
                taken += 1
                assert nbins <= dd.MAX_BINS and (eff * ((1 << n) - 1)).bit_length() <= nbins - 1, (A, n, h)
    assert taken > 5000 and refused > 1000


@pytest.mark.parametrize("n", [8, 16, 24, 32, 40, 48])
def test_sampled_weights_fit(lib, n):
    parity = 4 if n < 16 else 5 if n < 32 else 6
    for mode in (dd.MODE_MONTE_CARLO, dd.MODE_GRID_1D):
        nbins, _, _ = dd.request_shape(dd.Request(dd.CODE_EXT_HAMMING, mode, 1, n, m=100003))
        assert n + parity <= nbins - 1
    assert accepted(dd.Request(dd.CODE_EXT_HAMMING, dd.MODE_MONTE_CARLO, 1, 4, m=100)) is None
