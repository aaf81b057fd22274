"""Points that are on no curve of the library: their multiples and sums follow the
group law of the curve y^2 = x^3 + b' that they are on, the same at every size of
a call, and no signature over them passes as one of the identity."""
import random

import pytest

pytestmark = pytest.mark.gpu

from weighted_bte_b200 import ops  # noqa: E402

P = 0x1A0111EA397FE69A4B1BA7B6434BACD764774B84F38512BF6730D2A0F6B0F6241EABFFFEB153FFFFB9FEFFFFFFFFAAAB
R = ops.R
X_ABS = 0xD201000000010000


class Fp:
    @staticmethod
    def mul(a, b):
        return a * b % P

    @staticmethod
    def sub(a, b):
        return (a - b) % P

    @staticmethod
    def inv(a):
        return pow(a, -1, P)


class Fp2:
    @staticmethod
    def mul(a, b):
        return ((a[0] * b[0] - a[1] * b[1]) % P, (a[0] * b[1] + a[1] * b[0]) % P)

    @staticmethod
    def sub(a, b):
        return ((a[0] - b[0]) % P, (a[1] - b[1]) % P)

    @staticmethod
    def inv(a):
        n = pow(a[0] * a[0] + a[1] * a[1], -1, P)
        return (a[0] * n % P, -a[1] * n % P)


def add(F, p, q):
    """Sum of affine points (None: the identity) of a curve y^2 = x^3 + b'."""
    if p is None or q is None:
        return q if p is None else p
    zero = F.sub(p[1], p[1])
    if p[0] == q[0]:
        if p[1] != q[1] or p[1] == zero:
            return None
        xx = F.mul(p[0], p[0])
        lam = F.mul(F.sub(xx, F.sub(F.sub(zero, xx), xx)), F.inv(F.sub(p[1], F.sub(zero, p[1]))))
    else:
        lam = F.mul(F.sub(q[1], p[1]), F.inv(F.sub(q[0], p[0])))
    x = F.sub(F.sub(F.mul(lam, lam), p[0]), q[0])
    return x, F.sub(F.mul(lam, F.sub(p[0], x)), p[1])


def multiple(F, p, s):
    acc = None
    for bit in bin(s)[2:]:
        acc = add(F, acc, acc)
        if bit == "1":
            acc = add(F, acc, p)
    return acc


def words(v):
    return (v * (1 << 384) % P).to_bytes(48, "little")


def encode(p, size):
    if p is None:
        return bytes(size)
    return b"".join(words(c) for v in p for c in (v if isinstance(v, tuple) else (v,)))


G1_OFF = [(5, 7), (11, 0), (P - 2, 3)]
G2_OFF = [((5, 1), (7, 2)), ((3, 0), (0, 9))]
SCALARS = [0, 1, 2, 3, R - 1, 0x1234567]


@pytest.mark.parametrize("n", [1, 4, 700, 4001, 9001, 40000])
def test_multiples(n):
    rng = random.Random(n)
    scalars = SCALARS + [rng.randrange(R) for _ in range(3)]
    want = [encode(multiple(Fp, G1_OFF[i % 3], s), 96) for i, s in enumerate(scalars)]
    pts = [encode(G1_OFF[i % 3], 96) for i in range(len(scalars))]
    tile = lambda v: (v * (n // len(v) + 1))[:n]  # noqa: E731
    assert ops.split(ops.g1_mul(b"".join(tile(pts)), tile(scalars)), 96) == tile(want)


@pytest.mark.parametrize("n", [5, 33, 700])
def test_sums_of_one_point(n):
    rng = random.Random(n)
    scalars = [rng.randrange(R) for _ in range(n)]
    for p in G1_OFF:
        assert bytes(ops.g1_msm(encode(p, 96) * n, scalars)) == encode(multiple(Fp, p, sum(scalars)), 96)
    for p in G2_OFF:
        assert bytes(ops.g2_msm(encode(p, 192) * n, scalars)) == encode(multiple(Fp2, p, sum(scalars)), 192)


@pytest.mark.parametrize("k", [1, 7, 1500, 4001, 40000])
def test_small_sums(k):
    """One term of a family: s = a + b |x|^2 acts as a on p and b on phi(p) + p."""
    rng = random.Random(k)
    scalars = [rng.randrange(R) for _ in range(2)]
    beta = next(b for b in (pow(g, (P - 1) // 3, P) for g in range(2, 20)) if b != 1)
    gen = ops.g1_mul_generator([1, X_ABS * X_ABS - 1])
    gx = int.from_bytes(bytes(gen)[:48], "little")
    if gx * beta % P != int.from_bytes(bytes(gen)[96:144], "little"):
        beta = beta * beta % P
    assert gx * beta % P == int.from_bytes(bytes(gen)[96:144], "little")
    want = []
    for p in G1_OFF:
        acc = None
        for s in scalars:
            b, a = divmod(s, X_ABS * X_ABS)
            image = add(Fp, (p[0] * beta % P, p[1]), p)
            acc = add(Fp, acc, add(Fp, multiple(Fp, p, a), multiple(Fp, image, b)))
        want.append(encode(acc, 96))
    order = [i % 3 for i in range(k)]
    pts = b"".join(encode(G1_OFF[i], 96) * 2 for i in order)
    got = ops.split(ops.msm_family(1, pts, 2 * k, [2 * i for i in range(k)], None, scalars, None, 1, 2), 96)
    assert got == [want[i] for i in order]


@pytest.mark.parametrize("n", [1, 5, 700, 4001, 30000])
def test_no_signature_of_a_point_off_the_curve(n):
    rng = random.Random(n)
    good = bytes(ops.g1_mul_generator([rng.randrange(R)]))
    X = [encode((11, 0), 96), encode((5, 7), 96), good, good]
    Rc = [good, good, encode((11, 0), 96), encode((5, 7), 96)]
    s = [rng.randrange(R) for _ in X]
    c = [2 * rng.randrange(R // 2) + 1 for _ in X]
    tile = lambda v: (v * (n // len(v) + 1))[:n]  # noqa: E731
    assert not ops.schnorr_verify(b"".join(tile(X)), b"".join(tile(Rc)), tile(s), tile(c)).any()
