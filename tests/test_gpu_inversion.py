"""Inversions by division steps through the entry points that use one each:
scalars where the result is a fraction, field values where a point leaves its
projective form."""
import random

import pytest

pytestmark = pytest.mark.gpu

from oracle import oracle as orc  # noqa: E402
from weighted_bte_b200 import ops  # noqa: E402

R = ops.R


@pytest.mark.parametrize("x", [1, 2, R - 1, R - 2, (R + 1) // 2, 1 << 254, (1 << 30) - 1, 1 << 30, 3 << 200])
def test_scalar_inverse_at_its_edges(x):
    # L_0(0) = -y / (x - y) and L_1(0) = -x / (y - x) for the points x and y
    y = random.Random(x).randrange(1, R)
    d = pow(x - y, -1, R)
    assert ops.lagrange_at_zero([x, y]) == [-y * d % R, x * d % R]


@pytest.mark.parametrize("s", [0, 1, 2, R - 1, 0xD201000000010000, 1 << 254])
def test_field_inverse_through_affine_conversion(s):
    rng = random.Random(s)
    t = rng.randrange(R)
    assert ops.split(ops.g1_mul(orc.g1_generator() * 2, [s, t]), 96) == orc.g1_mul_many(orc.g1_generator(), [s, t])
    assert ops.split(ops.g2_mul(orc.g2_generator() * 2, [s, t]), 192) == orc.g2_mul_many(orc.g2_generator(), [s, t])
