"""Quad kernels (four places a point, one lane each in G1 and two in G2) at the
edges of their launches and at the special cases of the group law."""
import random

import pytest

pytestmark = pytest.mark.gpu

from oracle import oracle as orc  # noqa: E402
from weighted_bte_b200 import _lib, ops  # noqa: E402

R = ops.R
G = {1: (96, orc.g1_generator, orc.g1_mul_many, orc.g1_neg, ops.g1_mul, ops.g1_msm, orc.g1_msm, ops.g1_ntt, orc.g1_ntt),
     2: (192, orc.g2_generator, orc.g2_mul_many, orc.g2_neg, ops.g2_mul, ops.g2_msm, orc.g2_msm, ops.g2_ntt, orc.g2_ntt)}


def _points(group, rng, n):
    size, gen, mul = G[group][:3]
    pts = mul(gen(), [rng.randrange(R) for _ in range(n)])
    return pts


@pytest.mark.parametrize("group", [1, 2])
@pytest.mark.parametrize("n", [1, 3, 4, 5, 8, 9, 17])
def test_single_multiples(group, n):
    size, _, omul, _, mul = G[group][:5]
    rng = random.Random(n)
    pts = _points(group, rng, n)
    sc = [rng.randrange(R) for _ in range(n)]
    for i, s in enumerate([0, 1, R - 1, 16, 1 << 254]):
        if i < n:
            sc[(3 * i + 1) % n] = s
    if n > 2:
        pts[2] = bytes(size)
    assert ops.split(mul(b"".join(pts), sc), size) == omul(pts, sc)


@pytest.mark.parametrize("group", [1, 2])
@pytest.mark.parametrize("k,n", [(1, 1), (1, 3), (3, 2), (5, 4), (9, 3)])
def test_small_families_with_special_points(group, k, n):
    """Equal points, a point and its negative, the identity: doublings and
    cancellations inside the sums."""
    size, _, _, neg = G[group][:4]
    rng = random.Random(10 * k + n)
    pts = _points(group, rng, k * n)
    if n > 1:
        pts[1] = pts[0]
        pts[-1] = neg(pts[-2])
    if k > 2:
        pts[n] = bytes(size)
    sc = [rng.randrange(R) for _ in range(n)]
    if n > 1:
        sc[1] = sc[0]
        sc[-1] = sc[-2]
    got = ops.split(ops.msm_family(group, b"".join(pts), k * n, [n * i for i in range(k)], None, sc, None, 1, n), size)
    assert got == [G[group][6](pts[n * i : n * (i + 1)], sc) for i in range(k)]


@pytest.mark.parametrize("group", [1, 2])
@pytest.mark.parametrize("n", [5, 33, 200])
def test_window_tails(group, n):
    rng = random.Random(n)
    pts = _points(group, rng, n)
    for sc in ([rng.randrange(R) for _ in range(n)], [1] + [0] * (n - 1), [0] * n):
        assert G[group][5](b"".join(pts), sc) == G[group][6](pts, sc)


@pytest.mark.parametrize("group", [1, 2])
@pytest.mark.parametrize("n", [2, 4, 16, 64])
def test_transform_stages(group, n):
    size = G[group][0]
    rng = random.Random(n)
    pts = _points(group, rng, n)
    pts[1] = pts[0]
    pts[-1] = bytes(size)
    ctx = ops.ctx()
    ctx.set_tuning(_lib.TUNE_NTT_JOINT, 0)
    try:
        for inv in (False, True):
            assert ops.split(G[group][7](b"".join(pts), inverse=inv), size) == G[group][8](pts, inverse=inv)
    finally:
        ctx.set_tuning(_lib.TUNE_NTT_JOINT, -1)


@pytest.mark.parametrize("n", [1, 2, 3, 9])
def test_schnorr_checks(n):
    rng = random.Random(n)
    r, k, c = ([rng.randrange(R) for _ in range(n)] for _ in range(3))
    k[0] = 0  # a zero commitment
    X = b"".join(orc.g1_mul_many(orc.g1_generator(), r))
    C = b"".join(orc.g1_mul_many(orc.g1_generator(), k))
    s = [(a + b * x) % R for a, b, x in zip(k, c, r)]
    assert ops.schnorr_verify(X, C, s, c).all()
    for i in range(n):
        bad = list(s)
        bad[i] = (bad[i] + 1) % R
        assert list(ops.schnorr_verify(X, C, bad, c)) == [j != i for j in range(n)]
