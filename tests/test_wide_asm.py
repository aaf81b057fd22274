"""The double-width sequences of csrc/field_asm.cuh (12 x 12-word products,
Montgomery reduction of signed 24-word sums, conditional subtractions) run by
the PTX interpreter against big-integer arithmetic, with the bounds that the
team arithmetic relies on."""
import random

import pytest

from test_field_asm import P, call, limbs, value

R384 = 1 << 384
EDGES = [0, 1, P - 1, P, 2 * P, 8 * P, R384 - 1]


@pytest.mark.parametrize("a", EDGES)
def test_wide_product(a):
    rng = random.Random(a)
    for b in EDGES + [rng.randrange(R384) for _ in range(8)]:
        assert value(call("fp_mul_wide", a=limbs(a, 12), b=limbs(b, 12))["r"]) == a * b


@pytest.mark.parametrize("lo,hi,shift", [(-16, 6, 2), (-14, 8, 2), (-5, 17, 1), (-4, 8, 1), (-3, 3, 1)])
def test_reduction_of_signed_sums(lo, hi, shift):
    """Sums in (lo p^2, hi p^2), shifted by shift * p 2^384, reduce below 4p."""
    rng = random.Random(lo)
    for t in [0, lo * P * P + 1, hi * P * P - 1, R384, -R384, P * R384] + [
            rng.randrange(lo * P * P, hi * P * P) for _ in range(40)]:
        if not lo * P * P < t < hi * P * P:
            continue
        w = limbs(t % (1 << 768), 24)
        add = {1: "fp_add_p", 2: "fp_add_2p"}[shift]
        w = w[:12] + call(add, a=w[12:])["r"]
        r = value(call("fp_redc", t=w)["r"])
        assert r < 4 * P
        r = call("fp_csub_p", a=call("fp_csub_2p", a=limbs(r, 12))["r"])["r"]
        assert value(r) == t * pow(R384, -1, P) % P


def test_wide_sums_wrap():
    rng = random.Random(3)
    for _ in range(40):
        a, b = rng.randrange(1 << 768), rng.randrange(1 << 768)
        assert value(call("wide_add", a=limbs(a, 24), b=limbs(b, 24))["r"]) == (a + b) % (1 << 768)
        assert value(call("wide_sub", a=limbs(a, 24), b=limbs(b, 24))["r"]) == (a - b) % (1 << 768)


def test_sum_of_two_products():
    rng = random.Random(5)
    ri = pow(R384, -1, P)
    for k in range(60):
        a, b, c, d = ([0, 1, P - 1, P][rng.randrange(4)] if k < 30 else rng.randrange(P) for _ in range(4))
        got = call("fp_mont_mul2", a=limbs(a, 12), b=limbs(b, 12), c=limbs(c, 12), d=limbs(d, 12))["r"]
        assert value(got) == (a * b + c * d) * ri % P


def test_small_multiples():
    rng = random.Random(6)
    for _ in range(40):
        a = rng.randrange(8 * P)
        r = call("fp_csub_4p", a=limbs(a, 12))["r"]
        assert value(r) == (a - 4 * P if a >= 4 * P else a)
        b = rng.randrange(P + 1)
        assert value(call("fp_p_minus", a=limbs(b, 12))["r"]) == P - b
        b = rng.randrange(3 * P + 1)
        assert value(call("fp_3p_minus", a=limbs(b, 12))["r"]) == 3 * P - b


def test_square():
    rng = random.Random(7)
    ri = pow(R384, -1, P)
    for a in [0, 1, P - 1, P, 2 * P - 1] + [rng.randrange(2 * P) for _ in range(40)]:
        assert value(call("fp_mont_sqr", a=limbs(a, 12))["r"]) == a * a * ri % P


@pytest.mark.parametrize("ka,kb", [(8, 1), (1, 8), (7, 1), (1, 7), (4, 2), (2, 4), (3, 3)])
def test_product_of_sums_without_reduction(ka, kb):
    """Factors below ka p and kb p with ka kb < 2^384 / p give a reduced product;
    the first factor plus p has to stay below 2^384 as well."""
    rng = random.Random(10 * ka + kb)
    ri = pow(R384, -1, P)
    for k in range(30):
        a = [ka * P - 1, ka * P - 2, 0, P][k % 4] if k < 8 else rng.randrange(ka * P)
        b = [kb * P - 1, kb * P - 1, P, kb * P - 3][k % 4] if k < 12 else rng.randrange(kb * P)
        assert value(call("fp_mont_mul", a=limbs(a, 12), b=limbs(b, 12))["r"]) == a * b * ri % P
