"""Arithmetic of the kernels that can be checked on the host, against exact rationals."""
import random
from fractions import Fraction


def test_quotient_from_a_reciprocal_is_the_division():
    """The element matrices' quotients by one determinant: the product with its reciprocal and one
    correction by the exact remainder gives the correctly rounded quotient, the divisors whose
    significand is all ones or nearly included (float() of a rational rounds to nearest even, as a fused
    multiply-add does).  The product alone does not."""
    rnd = random.Random(1)
    uncorrected = 0
    for t in range(12000):
        if t % 3 == 0:
            a, b = (rnd.uniform(-1, 1) * 10.0 ** rnd.uniform(-8, 8) for _ in range(2))
        elif t % 3 == 1:
            a, b = float(rnd.getrandbits(53)), float(rnd.getrandbits(53) | 1)
        else:
            a, b = float(rnd.getrandbits(53)), float((1 << 53) - 1 - 2 * rnd.getrandbits(3))
        r = 1.0 / b
        q = a * r
        remainder = float(Fraction(a) - Fraction(q) * Fraction(b))
        assert float(Fraction(q) + Fraction(remainder) * Fraction(r)) == a / b, (a, b)
        uncorrected += q != a / b
    assert uncorrected > 1000
