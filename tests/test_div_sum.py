"""The FP64 collision divides by the reference's lattice constants through
div_sum (csrc/lbrb_internal.cuh): q0 = RN(x * RN(1/c)), r = fma(-q0, c, x),
result = fma(r, RN(1/c), q0) -- div_const without the choice that keeps the
sign of a zero.  Restated with exact rational arithmetic: the IEEE quotient for
every non-zero operand, and a zero for a zero."""
import random

from tests.test_div_const import DIVISORS, bits, div_const, fma, operands


def div_sum(x: float, c: float, rc: float) -> float:
    q0 = x * rc
    return fma(fma(-q0, c, x), rc, q0)


def test_div_sum_is_the_ieee_quotient():
    rng = random.Random(23)
    for name, c in DIVISORS.items():
        rc = 1.0 / c
        for x in operands(c, rng, 10000):
            got = div_sum(x, c, rc)
            if x == 0.0:
                assert got == 0.0
            else:
                assert bits(got) == bits(x / c) == bits(div_const(x, c, rc)), (name, x)
