"""The FP64 shortcuts of the reflection and of the entry formula round like the
operations they replace: quotients by a shared reciprocal, and reciprocal and
square root of numbers within 2^-30 of one (ehss_internal.cuh: quotient,
rcp_near_one, sqrt_near_one).  Every operation is replayed with exact rational
arithmetic rounded once to the nearest double."""
import math
import random
from fractions import Fraction as Q

import pytest


def rn(x):
    return float(x)                       # Fraction to float rounds to nearest, ties to even


def fma(a, b, c):
    return rn(Q(a) * Q(b) + Q(c))


def quotient(a, b, y):
    if a == 0.:
        return a * y
    w = rn(Q(fma(-b, y, 1.0)) * Q(y))
    q0 = fma(a, y, rn(Q(a) * Q(w)))
    return fma(fma(-b, q0, a), y, q0)


def rcp_near_one(b):
    return fma(1.0 - b, 1.0 + 2.0 ** -30, 1.0)


def sqrt_near_one(b):
    e = b - 1.0
    return fma(e, 0.5 + 2.0 ** -31 if e < 0 else 0.5 - 2.0 ** -31, 1.0)


def _mantissas(rng, n):
    for k in range(n):
        m = rng.getrandbits(52)
        if k % 4 == 1:
            m = (1 << 52) - 1 - rng.getrandbits(4)
        if k % 4 == 2:
            m = rng.getrandbits(4)
        yield 1.0 + m * 2.0 ** -52


def test_quotients_by_a_shared_reciprocal():
    rng = random.Random(1)
    for a, b in zip(_mantissas(rng, 40000), _mantissas(random.Random(2), 40000)):
        a, b = math.ldexp(a, rng.randint(-40, 40)) * rng.choice((1, -1)), math.ldexp(b, rng.randint(-8, 8))
        assert quotient(a, b, rn(1 / Q(b))) == a / b


def test_zero_numerators():
    for b in (.5, 1., 3.):
        for a in (0., -0.):
            assert math.copysign(1., quotient(a, b, 1 / b)) == math.copysign(1., a / b)
    assert math.isnan(quotient(0., 0., math.inf))          # a hit point that rounds onto its centre


@pytest.mark.parametrize('top', [64, 2 ** 22])
def test_near_one(top):
    rng = random.Random(top)
    offsets = range(-64, 65) if top == 64 else (rng.randint(-top + 1, top - 1) for _ in range(30000))
    for k in offsets:
        b = 1.0 + k * 2.0 ** (-52 if k > 0 else -53)
        assert abs(b - 1.0) <= 2.0 ** -30
        assert rcp_near_one(b) == 1.0 / b
        assert sqrt_near_one(b) == math.sqrt(b)
        a = rng.uniform(-3., 3.)
        assert quotient(a, b, rcp_near_one(b)) == a / b
