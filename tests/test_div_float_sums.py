"""The divergence's sums at the two finest depths: three floats by error-free additions stand in for a
sequential double sum (csrc/rhs.cu FloatSum3), restated here in float32 and compared with that sum."""
import numpy as np
import pytest

F = np.float32


def _float_sum3(terms):
    h = l = m = T = np.zeros(terms.shape[0], F)
    least = np.full(terms.shape[0], 0xFFFFFFFF, np.uint32)
    for k in range(terms.shape[1]):
        t = np.ascontiguousarray(terms[:, k])
        s = h + t
        a = s - h
        e = (h - (s - a)) + (t - a)
        q = l + e
        b = q - l
        m = m + ((l - (q - b)) + (e - b))
        h, l = s, q
        T = T + np.abs(t)
        least = np.minimum(least, (t.view(np.uint32) & np.uint32(0x7FFFFFFF)) - np.uint32(1))
    v = h.astype(np.float64) + (l.astype(np.float64) + m.astype(np.float64))
    d = T.astype(np.float64) * 2.0 ** -44
    f = (v - d).astype(F)
    eT = (T.view(np.uint32) >> 23).astype(int)
    en = np.maximum(((least + np.uint32(1)) >> 23).astype(int), 1)
    same = f == (v + d).astype(F)
    return np.where(same, f, v.astype(F)), same | ((eT < 255) & (eT - en <= 28))


def _double_sum(terms):
    d = np.zeros(terms.shape[0])
    for k in range(terms.shape[1]):
        d = d + terms[:, k].astype(np.float64)
    return d.astype(F)


@pytest.mark.parametrize("n", [1, 2, 27, 216])
@pytest.mark.parametrize("spread", [0, 12, 40, 100])
def test_equals_the_double_sum_wherever_it_says_so(n, spread):
    rng = np.random.default_rng(1000 * n + spread)
    rows = 20_000
    t = (rng.standard_normal((rows, n)) * np.exp2(rng.uniform(-spread, 0, (rows, n)))).astype(F)
    t[rng.random((rows, n)) < 0.1] = 0
    with np.errstate(all="ignore"):
        f, sure = _float_sum3(t)
        assert np.array_equal(f[sure], _double_sum(t)[sure])
    assert sure.mean() > 0.999


def test_cancellation_ties_and_non_finite_values_are_not_claimed():
    big = F(2.0 ** 30)
    rows = [
        [big, F(1e-20), -big] + [F(0)] * 24,             # what is left is far below the terms
        [F(1), F(2.0 ** -24), F(2.0 ** -60)] + [F(0)] * 24,   # just above a tie of the float rounding
        [F(np.inf), F(1)] + [F(0)] * 25,
        [F(np.nan)] + [F(0)] * 26,
        [F(3e38), F(3e38), F(-3e38)] + [F(0)] * 24,      # overflows in float, not in double
        [F(0)] * 27,
    ]
    t = np.array(rows, F)
    with np.errstate(all="ignore"):
        f, sure = _float_sum3(t)
        ref = _double_sum(t)
    assert list(sure) == [False, False, False, False, False, True]
    assert f[5] == 0 and ref[4] == F(3e38)
