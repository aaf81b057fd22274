"""MSMs longer than a plan's full complement of segments, over known multiples of
the generator: the sum is one multiple of it."""
import random

import pytest

pytestmark = pytest.mark.gpu

from oracle import oracle as orc  # noqa: E402
from weighted_bte_b200 import ops  # noqa: E402


@pytest.mark.parametrize("n", [100003, (1 << 17) + 3, 1 << 18])
def test_sums_of_multiples(n):
    rng = random.Random(n)
    u = [rng.randrange(ops.R) for _ in range(509)]
    s = [rng.randrange(ops.R) for _ in range(n)]
    s[0], s[1], s[2], s[n - 1] = 0, 1, ops.R - 1, ops.R - 1
    total = sum(a * u[i % len(u)] for i, a in enumerate(s)) % ops.R
    tile = lambda b, size: (b * (n // len(u) + 1))[: size * n]  # noqa: E731
    sc = ops.scalars_bytes(s)
    assert bytes(ops.g1_msm(tile(bytes(ops.g1_mul_generator(u)), 96), sc)) == orc.g1_mul_many(orc.g1_generator(), [total])[0]
    assert bytes(ops.g2_msm(tile(bytes(ops.g2_mul_generator(u)), 192), sc)) == orc.g2_mul_many(orc.g2_generator(), [total])[0]
