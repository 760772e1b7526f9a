"""The last step of div_rn (harm_phys.cuh) in exact rational arithmetic on the
CPU: with y = RN(1/b), a faithful quotient q and its exact remainder r = a - b q,
RN(q + r y) is the IEEE quotient (Markstein).  Fed both neighbours of a/b, near
rounding midpoints and around powers of two; and the whole routine.  The device
routine itself is compared with the device's division in test_divrn.py."""
import random
from fractions import Fraction

import pytest

from test_divrn import bits, fma, from_bits, rand_double


def last_step(a, b, y, q):
    return fma(fma(-q, b, a), y, q)


def cases(n, seed):
    rng = random.Random(seed)
    for t in range(n):
        eb = rng.randint(-60, 60)
        b = from_bits(((eb + 1023) << 52) | (0xFFFFFFFFFFFFF - t % 3)) if t % 7 == 0 else rand_double(rng, eb, eb, False)
        if t % 3 == 0:
            # a/b next to the midpoint of two doubles
            q = rand_double(rng, -60, 60)
            h = from_bits((((bits(q) >> 52) & 0x7FF) - 53) << 52)
            a = float(Fraction(b) * (Fraction(q) + Fraction(h) * rng.choice((1, -1))))
        elif t % 3 == 1:
            z = Fraction(2) ** rng.randint(-50, 50) * rng.choice((1, -1))
            a = float(Fraction(b) * z * (1 + Fraction(rng.randint(-8, 8), 2 ** 53)))
        else:
            a = rand_double(rng, -790, 790)
        yield a, b


@pytest.mark.parametrize("seed", [1, 2])
def test_fma_last_step_rounds_correctly_from_either_neighbour(seed):
    for a, b in cases(30000, seed):
        want, z = a / b, Fraction(a) / Fraction(b)
        y = 1. / b
        lo = want if Fraction(want) <= z else from_bits(bits(want) - 1 if want > 0 else bits(want) + 1)
        hi = want if Fraction(want) >= z else from_bits(bits(want) + 1 if want > 0 else bits(want) - 1)
        for q in (lo, hi):
            assert bits(last_step(a, b, y, q)) == bits(want), (a, b, q)
        q = a * y
        q = fma(fma(-q, b, a), y, q)
        assert bits(last_step(a, b, y, q)) == bits(want), (a, b)
