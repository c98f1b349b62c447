"""The solvers' warp sum: the lanes' doubles aligned to the largest exponent as 58-bit integers and added
as integers, restated here step by step (csrc/cg_common.cuh warp_sum, warp_sum_aligned)."""
import struct
from fractions import Fraction

import numpy as np
import pytest


def _bits(v):
    return struct.unpack("<Q", struct.pack("<d", v))[0]


def _warp_sum(vals):
    es = [(_bits(v) >> 52) & 0x7FF for v in vals]
    emax = max(es)
    assert 64 <= emax < 0x7FF      # other exponents take the butterfly of doubles
    S = 0
    for v, e in zip(vals, es):
        m = (_bits(v) & ((1 << 52) - 1)) | ((1 << 52) if e else 0)
        x = (m << 5) >> min(emax - e, 63)
        x = -x if _bits(v) >> 63 else x
        # limbs of 24, 24 and 16 bits: 32 lanes' sums fit 32-bit integers
        lo, mid, hi = x & 0xFFFFFF, (x >> 24) & 0xFFFFFF, x >> 48
        assert abs(hi) < 2 ** 15
        S += (hi << 48) + (mid << 24) + lo
    assert abs(S) < 2 ** 63
    if S == 0:
        return 0.0
    q = emax - 1080
    u = abs(S)
    lz = 64 - u.bit_length()
    u <<= lz
    bits = ((1023 + 63 - lz + q) << 52) + ((u >> 11) & ((1 << 52) - 1)) + ((u >> 10) & 1)
    return struct.unpack("<d", struct.pack("<Q", bits | ((1 << 63) if S < 0 else 0)))[0]


@pytest.mark.parametrize("seed,spread,lanes", [(0, 0, 32), (1, 10, 32), (2, 60, 32), (3, 30, 8), (4, 200, 32), (5, 1, 1)])
def test_aligned_sum_is_within_a_double_rounding(seed, spread, lanes):
    rng = np.random.default_rng(seed)
    for _ in range(200):
        v = [float(x) for x in rng.standard_normal(lanes) * np.exp2(rng.uniform(-spread, spread, lanes))] + [0.0] * (32 - lanes)
        exact = sum((Fraction(x) for x in v), Fraction(0))
        big = max(abs(Fraction(x)) for x in v)
        err = abs(Fraction(_warp_sum(v)) - exact)
        # 32 lanes each truncated below 2^-57 of the largest value's power of two, and one rounding of the sum
        assert err <= 32 * big * Fraction(1, 2 ** 57) + abs(exact) * Fraction(1, 2 ** 53)


def test_exact_cases():
    assert _warp_sum([1.0, -1.0] + [0.0] * 30) == 0.0
    assert _warp_sum([float(2 ** 53 - 1)] + [1.0] + [0.0] * 30) == float(2 ** 53)
    assert _warp_sum([1.5] * 32) == 48.0
