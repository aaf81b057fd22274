"""G1 chains on eight lanes a point and on quads, on both sides of the line
between them, against the oracle."""
import random

import pytest

pytestmark = pytest.mark.gpu

from oracle import oracle as orc  # noqa: E402
from weighted_bte_b200 import ops  # noqa: E402

R = ops.R


def _points(rng, n):
    return orc.g1_mul_many(orc.g1_generator(), [rng.randrange(R) for _ in range(n)])


@pytest.mark.parametrize("n", [1, 3, 4, 5, 1000, 5790, 5803, 9001])
def test_multiples(n):
    rng = random.Random(n)
    pts = _points(rng, 9)
    pts[4] = bytes(96)
    sc = [rng.randrange(R) for _ in range(9)]
    sc[0], sc[5], sc[6] = 0, 1, R - 1
    want = orc.g1_mul_many(pts, sc)
    tile = lambda v: (v * (n // 9 + 1))[:n]  # noqa: E731
    assert ops.split(ops.g1_mul(b"".join(tile(pts)), tile(sc)), 96) == tile(want)


@pytest.mark.parametrize("n", [2, 8, 64, 512, 2048])
def test_transforms(n):
    rng = random.Random(n)
    pts = _points(rng, n)
    pts[1] = pts[0]
    if n > 4:
        pts[3] = bytes(96)
    for inverse in (False, True):
        assert ops.split(ops.g1_ntt(b"".join(pts), inverse=inverse), 96) == orc.g1_ntt(pts, inverse=inverse)


@pytest.mark.parametrize("k", [1, 7, 1500, 4001])
def test_small_sums_that_double_and_cancel(k):
    rng = random.Random(k)
    a, b = _points(rng, 2)
    kinds = [[a, a], [a, orc.g1_neg(a)], [a, b], [bytes(96), b], [bytes(96), bytes(96)]]
    s = rng.randrange(R)
    for sc in ([s, s], [s, R - s], [1, 1]):
        want = [orc.g1_msm(p, sc) for p in kinds]
        order = [i % 5 for i in range(k)]
        pts = b"".join(p for i in order for p in kinds[i])
        got = ops.split(ops.msm_family(1, pts, 2 * k, [2 * i for i in range(k)], None, sc, None, 1, 2), 96)
        assert got == [want[i] for i in order]


@pytest.mark.parametrize("n", [1, 2, 40, 300])
def test_msm_of_special_points(n):
    """Window sums that are the identity, equal or opposite in the Horner tail."""
    rng = random.Random(n)
    a = _points(rng, 1)[0]
    pts = [a if i % 3 else orc.g1_neg(a) for i in range(n)]
    for sc in ([1] * n, [R - 1] * n, [(1 << (i % 254)) for i in range(n)], [0] * n):
        assert ops.g1_msm(b"".join(pts), sc) == orc.g1_msm(pts, sc)


@pytest.mark.parametrize("group", [1, 2])
@pytest.mark.parametrize("n", [1, 5, 3000, 5000, 12001, 40000])
def test_generator_multiples(group, n):
    """One to eight lanes (pairs in G2) per multiple."""
    rng = random.Random(n)
    sc = [0, 1, R - 1, 1 << 248, 255] + [rng.randrange(R) for _ in range(4)]
    mul, gen, fast, size = ((orc.g1_mul_many, orc.g1_generator, ops.g1_mul_generator, 96),
                            (orc.g2_mul_many, orc.g2_generator, ops.g2_mul_generator, 192))[group - 1]
    tile = lambda v: (v * (n // 9 + 1))[:n]  # noqa: E731
    assert ops.split(fast(tile(sc)), size) == tile(mul(gen(), sc))
