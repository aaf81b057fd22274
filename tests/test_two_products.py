"""The sum of two products with one reduction over its whole domain: first factors up
to p, second factors whose sum fits 384 bits, unreduced sums below 4p among them."""
import random

import pytest

from test_field_asm import P, call, limbs, value

R384 = 1 << 384
FIRST = [0, 1, P - 1, P]
SECOND = [0, 1, P, 2 * P - 1, 4 * P - 2, 4 * P - 1]


def _check(a, b, c, d):
    got = call("fp_mont_mul2", a=limbs(a, 12), b=limbs(b, 12), c=limbs(c, 12), d=limbs(d, 12))["r"]
    assert value(got) == (a * b + c * d) * pow(R384, -1, P) % P


@pytest.mark.parametrize("a", FIRST)
def test_edges(a):
    for c in (P - 1, P):
        for b in SECOND:
            for d in SECOND:
                _check(a, b, c, d)
    for b, d in ((R384 - 1, 1), (R384 - P, P), (R384 // 2, R384 // 2)):
        _check(a, b, P, d)


def test_random_factors():
    rng = random.Random(11)
    for _ in range(60):
        _check(rng.randrange(P + 1), rng.randrange(4 * P), rng.randrange(P + 1), rng.randrange(4 * P))
