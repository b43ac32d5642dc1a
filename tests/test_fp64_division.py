"""Division by a known divisor (div_known of the FP64 kernels) restated on the
CPU with exact rational arithmetic: two-part reciprocal, one product, three
fused multiply-adds -- equal to the correctly rounded quotient for random
operands and for the ones hardest to round (quotients next to a midpoint,
divisors next to a power of two)."""
from fractions import Fraction
import random
import struct

import pytest


def fma(a, b, c):
    """a * b + c rounded once (Fraction -> float rounds to nearest even)."""
    return float(Fraction(a) * Fraction(b) + Fraction(c))


def recip(m):
    yh = float(1 / Fraction(m))
    return yh, fma(-yh, m, 1.0) * yh


def div_known(x, m):
    yh, yl = recip(m)
    q0 = fma(x, yh, x * yl)
    return fma(fma(-q0, m, x), yh, q0)


def mantissas(kind, rng):
    one = 1 << 52
    if kind == "random":
        return rng.randrange(one, 2 * one), rng.randrange(one, 2 * one)
    if kind == "edge":  # mantissas of few set or few clear low bits
        pick = lambda: rng.choice([one + rng.randrange(4), 2 * one - 1 - rng.randrange(4), one + (1 << rng.randrange(52))])  # noqa: E731
        return pick(), pick()
    # quotients next to a midpoint of two doubles: x = (q + 1/2) m + small,
    # solved for the smallest remainders modulo the divisor (odd m)
    m = rng.randrange(one, 2 * one) | 1
    r = rng.choice([-3, -1, 1, 3])
    for shift in (53, 54):
        # 2^shift x = m (2 q + 1) + r  =>  (2 q + 1) = -r / m  (mod 2^shift)
        odd = (-r * pow(m, -1, 1 << shift)) % (1 << shift)
        x = (m * odd + r) >> shift
        if odd & 1 and one <= x < 2 * one:
            return x, m
    return rng.randrange(one, 2 * one), m


@pytest.mark.parametrize("kind", ["random", "edge", "midpoint"])
def test_equals_division(kind):
    rng = random.Random(20)
    for _ in range(6000):
        a, b = mantissas(kind, rng)
        x = float(a) * 2.0 ** rng.randrange(-400, 400) * rng.choice([1.0, -1.0])
        m = float(b) * 2.0 ** rng.randrange(-300, 300)
        q = div_known(x, m)
        assert struct.pack("d", q) == struct.pack("d", x / m), (x.hex(), m.hex())


def test_zero_dividend():
    for m in (1.0, 3.7e-12, 8.1e20):
        assert div_known(0.0, m) == 0.0 and div_known(-0.0, m) == 0.0
