"""The integer-pipe product, reciprocal and divisions that stand in for FP64 instructions, on the GPU against IEEE
arithmetic, bit for bit: any bit patterns, results next to a rounding boundary, powers of two, the ends of the range."""
import numpy as np
import pytest

import mdz_rheo as R

pytestmark = pytest.mark.gpu


def bits(x):
    return np.ascontiguousarray(x, np.float64).view(np.uint64)


def same(got, want):
    return (bits(got) == bits(want)) | (np.isnan(got) & np.isnan(want))


def patterns(rng, n):
    """Random doubles: every exponent, exponents near 1, short significands, significands at the ends of a binade."""
    x = rng.integers(0, 1 << 64, n, dtype=np.uint64)
    x[1::4] = (x[1::4] & np.uint64(0x800fffffffffffff)) | ((np.uint64(990) + x[1::4] % np.uint64(64)) << np.uint64(52))
    x[2::4] &= np.uint64(0xfffffffffc000000)
    ends = x[3::8]
    ends[:] = (ends & np.uint64(0xfff0000000000000)) | (ends % np.uint64(200))
    x[7::16] |= np.uint64(0x000fffffffffff00)
    special = bits([0.0, -0.0, 1.0, -1.0, 2.0 ** 1000, 2.0 ** -1000, 2.0 ** 1001, 2.0 ** -1001, 5e-324, -1e-310, 1.7e308, np.inf,
                    -np.inf, np.nan])
    x[:special.size] = special
    return x.view(np.float64)


def reciprocal_ties(rng, n):
    """Significands m whose reciprocal 2^104 / m lies within a few parts in 2^64 of half a unit: from the wanted
    quotient (an odd multiple of a half), m is the nearest integer."""
    half = (rng.integers(1 << 52, 1 << 53, n).astype(object) * 2 + 1)
    m = [(1 << 106) // int(h) for h in half]
    m = np.array([v if (1 << 52) <= v < (1 << 53) else (1 << 52) for v in m], dtype=np.uint64)
    return ((m & np.uint64((1 << 52) - 1)) | (np.uint64(1023) << np.uint64(52))).view(np.float64)


def test_against_ieee():
    rng = np.random.default_rng(17)
    n = 2_000_000
    a, b = patterns(rng, n), patterns(rng, n)
    rng.shuffle(b)
    ties = reciprocal_ties(rng, 50_000)
    a = np.concatenate([a, ties, -ties * 2.0 ** 40])
    near = (np.int64(0x3ff0000000000000) + rng.integers(-40, 24, a.size - n // 2)).view(np.float64)
    b = np.concatenate([b[:n // 2], near])  # any divisor, then divisors near 1
    out = R.fx_pair_selftest(a, b)
    with np.errstate(all="ignore"):
        want = {"product": a * b, "reciprocal": 1.0 / a, "division by a weight sum": a / b,
                "division, divisor formed on the device": a / b}
    for (name, w), got in zip(want.items(), out[2:]):
        bad = ~same(got, w)
        assert not bad.any(), (name, bad.sum(), a[bad][:3], b[bad][:3])
