"""Teams of twelve lanes take over from teams of six where a launch has few
values: the same outputs on both sides of the line, against the oracle."""
import random

import pytest

pytestmark = pytest.mark.gpu

from oracle import oracle as orc  # noqa: E402
from weighted_bte_b200 import ops  # noqa: E402

KINDS = 7  # distinct values of each input, repeated to the launch's size


def _rs(rng, n):
    return [rng.randrange(ops.R) for _ in range(n)]


def _tile(vals, n):
    return (vals * (n // len(vals) + 1))[:n]


@pytest.mark.parametrize("n", [3, 1184, 1185, 2961, 6001])
def test_pairings_powers_and_products(n):
    rng = random.Random(n)
    p = orc.g1_mul_many(orc.g1_generator(), _rs(rng, KINDS))
    q = orc.g2_mul_many(orc.g2_generator(), _rs(rng, KINDS))
    p[2], q[1] = bytes(96), bytes(192)
    gt = [orc.pairing(a, b) for a, b in zip(p, q)]
    P, Q = b"".join(_tile(p, n)), b"".join(_tile(q, n))
    expect = _tile(gt, n)
    f = ops.miller_loop(P, Q)
    assert ops.split(ops.final_exp(f), 576) == expect
    g = ops.miller_loop_lines(ops.prepare_lines(Q), P)
    assert ops.split(ops.final_exp(ops.final_exp(g, mode=1), mode=2), 576) == expect
    sc = _rs(rng, KINDS)
    powers = [orc.gt_pow_many(v, [s])[0] for v, s in zip(gt, sc)]
    assert ops.split(ops.gt_pow(b"".join(expect), _tile(sc, n)), 576) == _tile(powers, n)
    products = [orc.fp12_mul(a, b) for a, b in zip(gt, powers)]
    assert ops.split(ops.fp12_mul(b"".join(expect), b"".join(_tile(powers, n))), 576) == _tile(products, n)


@pytest.mark.parametrize("n,count", [(8, 7), (8, 147), (8, 149), (16, 300)])
def test_transforms(n, count):
    rng = random.Random(n * 1000 + count)
    arrays = [orc.gt_pow_many(orc.pairing(orc.g1_generator(), orc.g2_generator()), _rs(rng, n)) for _ in range(KINDS)]
    for inv in (False, True):
        got = ops.split(ops.gt_ntt_many(b"".join(v for a in _tile(arrays, count) for v in a), n, inverse=inv), 576)
        want = [orc.gt_ntt(a, inverse=inv) for a in arrays]
        assert got == [v for a in _tile(want, count) for v in a]


@pytest.mark.parametrize("n", [1, 2, 3, 7, 1184])
def test_torus_encodings_of_few_values(n):
    """Against one thread per value, which longer calls take."""
    rng = random.Random(n)
    one = orc.fp12_one()
    kinds = orc.gt_pow_many(orc.pairing(orc.g1_generator(), orc.g2_generator()), _rs(rng, 4))
    kinds += [one, bytes(288) + kinds[0][288:], kinds[1][:288] + bytes(288), bytes(576)]
    many = 1500
    want = ops.split(ops.gt_compress(b"".join(_tile(kinds, many)), many), 289)
    assert ops.split(ops.gt_compress(b"".join(_tile(kinds, n)), n), 289) == want[:n]
    assert want[4] == bytes(289)
