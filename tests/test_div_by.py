"""The kernels' quotients by fixed divisors (div_by, mg_div): a product with the correctly
rounded reciprocal and two residual corrections must round like the division. Emulated with
exact rationals; the roundings are the operations' own."""
import random
from fractions import Fraction

import pytest


def rn(x: Fraction, bits: int) -> Fraction:
    """x rounded to `bits` binary digits, ties to even (exponents unbounded)."""
    if x == 0:
        return x
    e = 0
    n, d = abs(x).numerator, abs(x).denominator
    e = n.bit_length() - d.bit_length() - bits
    while True:
        q = abs(x) / Fraction(2) ** e
        if q >= 2 ** bits:
            e += 1
        elif q < 2 ** (bits - 1):
            e -= 1
        else:
            break
    f = q.numerator // q.denominator
    r = q - f
    if r > Fraction(1, 2) or (r == Fraction(1, 2) and f & 1):
        f += 1
    return (1 if x > 0 else -1) * f * Fraction(2) ** e


@pytest.mark.parametrize("bits", [24, 53])
def test_corrected_quotient_is_the_rounded_quotient(bits):
    rng = random.Random(bits)
    top = 2 ** bits
    special = [top // 2, top // 2 + 1, top - 1, top - 2, (top // 3) | 1]
    for k in range(4000):
        n = Fraction(rng.choice(special) if k % 3 == 0 else rng.randrange(top // 2, top)) * Fraction(2) ** rng.randint(-9, 9)
        d = Fraction(rng.choice(special) if k % 4 == 0 else rng.randrange(top // 2, top)) * Fraction(2) ** rng.randint(-9, 9)
        n = -n if k & 1 else n
        y = rn(1 / d, bits)
        q = rn(n * y, bits)
        for _ in range(2):
            q = rn(q + rn(n - d * q, bits) * y, bits)
        assert q == rn(n / d, bits), (n, d)
