"""The solvers' warp sums (csrc/cg_common.cuh warp_sum) as the GPU forms them, of doubles and of compensated float
pairs, against exact sums: exponents that spread more than the aligned integers hold, subnormal floats, zeros,
cancellation, and values that are not finite or too small for the alignment, which take the butterfly.

Bounds: aligned to the largest exponent, a double drops less than 2^-57 of the largest value's power of two and each
float of a pair less than 2^-56, 32 and 64 of them at most; the sum is rounded once."""
import ctypes
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

from conftest import REPO

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def sums(tmp_path_factory):
    from poissonrecon_gpu_gb300 import builder
    lib = str(tmp_path_factory.mktemp("warp") / "warp_sums.so")
    subprocess.run([builder.NVCC] + builder.CU_FLAGS + ["-shared", os.path.join(REPO, "tests", "cpp", "warp_sums.cu"), "-o", lib],
                   check=True)
    L = ctypes.CDLL(lib)
    L.warp_sums.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.c_void_p]

    def run(v):
        v = np.ascontiguousarray(v)
        out = np.empty(len(v))
        assert L.warp_sums(v.ctypes.data, len(v), int(v.dtype == np.float32), out.ctypes.data) == 0
        return out
    return run


def _check(got, rows, drop):
    for s, row in zip(got, rows):
        v = [Fraction(float(x)) for x in np.ravel(row)]
        exact, big = sum(v, Fraction(0)), max(abs(x) for x in v)
        # the largest value's power of two, from its exponent
        top = Fraction(2) ** (int(np.frexp(float(big))[1]) - 1) if big else Fraction(0)
        assert abs(Fraction(float(s)) - exact) <= drop * top + abs(exact) / 2 ** 53


@pytest.mark.parametrize("spread", [0, 3, 20, 60, 300, 1000])
@pytest.mark.parametrize("lanes", [1, 8, 31, 32])
def test_doubles(sums, spread, lanes):
    rng = np.random.default_rng(1000 * spread + lanes)
    v = rng.standard_normal((300, 32)) * np.exp2(rng.uniform(-spread, min(spread, 900), (300, 32)))
    v[:, lanes:] = 0.0
    v[::7] = np.abs(v[::7])
    _check(sums(v), v, Fraction(32, 2 ** 57))


@pytest.mark.parametrize("scale", [-149, -140, -126, -100, 0, 60, 122])
@pytest.mark.parametrize("spread", [0, 10, 40, 120])
def test_pairs(sums, scale, spread):
    rng = np.random.default_rng(1000 * spread + scale + 200)
    with np.errstate(all="ignore"):
        h = (rng.standard_normal((300, 32)) * np.exp2(scale - rng.uniform(0, spread, (300, 32)))).astype(np.float32)
        l = (rng.uniform(-1, 1, (300, 32)) * np.abs(h) * 2.0 ** -24).astype(np.float32)
    h[::5, 3:] = 0.0
    h[::7] = np.abs(h[::7])
    h[::11, 16:] = -h[::11, :16]
    v = np.stack([h, l], 2)
    _check(sums(v), v, Fraction(64, 2 ** 56))


def test_exact_and_special_values(sums):
    zero = np.zeros(32)
    tiny = np.full(32, 5e-324)
    rows = np.array([zero, -zero, tiny, np.r_[1.0, -1.0, zero[2:]], np.full(32, 1.5), np.r_[2.0 ** 53 - 1, 1.0, zero[2:]],
                     np.r_[np.inf, np.ones(31)], np.r_[np.inf, -np.inf, zero[2:]], np.r_[np.nan, np.ones(31)],
                     np.r_[2.0 ** 1023, 2.0 ** 1023, zero[2:]], np.full(32, 1.7e308), np.full(32, 2.0 ** 1018),
                     np.r_[np.full(16, 1.7e308), np.full(16, -1.7e308)]])
    got = sums(rows)
    want = [0, 0, 32 * 5e-324, 0, 48, 2.0 ** 53, np.inf, np.nan, np.nan, np.inf, np.inf, 2.0 ** 1023, 0]
    assert np.array_equal(got, want, equal_nan=True)
    small = np.float32(1e-45)
    pairs = np.zeros((5, 32, 2), np.float32)
    pairs[1, :, 0] = small
    pairs[2, 0, 0], pairs[2, 1, 0] = np.inf, 1
    pairs[3, 0, 0], pairs[3, 1, 0] = np.inf, -np.inf
    pairs[4, 7, 1] = np.nan
    got = sums(pairs)
    assert np.array_equal(got, [0, 32 * float(small), np.inf, np.nan, np.nan], equal_nan=True)
