"""Two shortcuts in the quantisation of a GEMV's columns (mmvq_mma.cuh, mv_quantize), restated in f32 arithmetic and compared with what they stand for: roundf by an addition and a
cut, and the quotient by 127 by the rounded reciprocal and one correction (Markstein's theorem)."""
import numpy as np
import pytest

F = np.float32
pytestmark = pytest.mark.skipif(np.finfo(np.longdouble).nmant < 63, reason="the fused multiply-add is restated in 64 bits of mantissa")


def test_rounding_half_away_from_zero_below_128():
    """Every float from 1/4 to 128; below, what is added leaves less than 3/4, which is cut to 0.  (Signs are symmetric.)"""
    assert F(0.25) + F(0.49999997) < 1
    for e in range(125, 134):  # exponents of 2^-2 .. 2^6
        x = (np.arange(1 << 23, dtype=np.uint32) | np.uint32(e << 23)).view(F)
        want = np.floor(x)
        want += x - want >= F(0.5)  # exact: x - floor(x) is a float
        assert np.array_equal(np.trunc(x + F(0.49999997)), want), e


def quotient(a):
    r = F(1) / F(127)
    q = (a * r).astype(F)
    rest = (np.float64(-127) * q.astype(np.float64) + a).astype(F)  # exact in 64 bits, and a float
    return (rest.astype(np.longdouble) * np.longdouble(r) + q.astype(np.longdouble)).astype(F)


def test_quotient_by_127():
    """Every mantissa; what lies between the limits of the shortcut (1e-25 and 1e38) is that times a power of two, denormals are far away: a sample at every exponent."""
    x = (np.arange(1 << 23, dtype=np.uint32) | np.uint32(127 << 23)).view(F)
    assert np.array_equal(quotient(x), x / F(127))
    rng = np.random.default_rng(0)
    for e in range(44, 254):
        x = (rng.integers(0, 1 << 23, 4096, dtype=np.uint32) | np.uint32(e << 23)).view(F)
        x = x[(x > 1e-25) & (x < 1e38)]
        assert np.array_equal(quotient(x), x / F(127)), e
