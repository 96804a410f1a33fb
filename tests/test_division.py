"""The three-operation division of the reference-precision kernels
(divided_by in stencil_common.cuh, Recip in sgs_kernels.cuh), restated with the
C library's fused multiply-add: its quotient against the division's, bit for
bit, for the literals and for awkward spacings, on random dividends and on
those whose quotients lie next to the middle of two doubles, where a wrong
rounding would show first."""
import ctypes
import ctypes.util
import math
import random
from fractions import Fraction

import pytest

LIBM = ctypes.CDLL(ctypes.util.find_library("m"))
LIBM.fma.restype = ctypes.c_double
LIBM.fma.argtypes = [ctypes.c_double] * 3
fma = LIBM.fma

DIVISORS = {
    "p00": 1e5, "234.5": 234.5, "third": 1.0 / 3.0, "500 m": 500.0, "20 km / 41": 20000.0 / 41, "333.3 m": 333.3,
    "below 512": math.nextafter(512.0, 0.0), "above 256": math.nextafter(256.0, 512.0),
    "3 ulp below 1024": 1024.0 - 3 * math.ulp(1000.0), "1.999": 1.9990234375 + 2.0 ** -40,
}


def _quotient(x, d):
    y = 1.0 / d
    q = x * y
    return fma(-fma(d, q, -x), y, q), q


def _next_to_middles(d):
    """Dividends x with 53 bits whose quotient x / d is as near to the middle
    of two doubles as any: 2^s x = +-r modulo d's odd part."""
    odd = d.as_integer_ratio()[0]
    odd //= odd & -odd
    out = []
    if odd < 3:
        return out
    for s in range(50, 56):
        inverse = pow(pow(2, s, odd), -1, odd)
        for r in (-5, -3, -2, -1, 1, 2, 3, 5):
            x = r * inverse % odd
            x += -(-max(0, 2 ** 52 - x) // odd) * odd
            if 2 ** 52 <= x < 2 ** 53:
                out.append(float(x))
    return out


@pytest.mark.parametrize("d", DIVISORS.values(), ids=DIVISORS)
def test_quotient_rounds_as_the_division(d):
    rng = random.Random(5)
    dividends = [rng.uniform(1, 2) * 2.0 ** rng.randint(-40, 40) for _ in range(20000)] + _next_to_middles(d)
    first = 0.0
    for x in dividends:
        for v in (x, -x):
            got, q = _quotient(v, d)
            assert got == v / d, (v, d)
        first = max(first, float(abs(Fraction(q) - Fraction(v) / Fraction(d)) / Fraction(math.ulp(got))))
    assert first <= 1.5  # the first quotient's error, in ulps


@pytest.mark.parametrize("d", [1e5, 500.0])
def test_zeros_keep_their_sign(d):
    """For positive divisors, the only ones that take this form (the closure's
    host check admits those within 2^+-60, the literals are positive)."""
    for x in (0.0, -0.0):
        assert math.copysign(1.0, _quotient(x, d)[0]) == math.copysign(1.0, x / d)
