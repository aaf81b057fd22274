"""Six-lane Fp12 kernels at the edges of their launches (five teams a warp,
four where a power is spread over several) against the oracle."""
import random

import pytest

pytestmark = pytest.mark.gpu

from oracle import oracle as orc  # noqa: E402
from weighted_bte_b200 import _lib, ops  # noqa: E402


def _rs(rng, n):
    return [rng.randrange(ops.R) for _ in range(n)]


@pytest.fixture(scope="module")
def base():
    return orc.pairing(orc.g1_generator(), orc.g2_generator())


@pytest.mark.parametrize("teams", [0, 1, 2, 4])
@pytest.mark.parametrize("n", [1, 4, 5, 6, 11])
def test_powers_and_products(base, n, teams):
    rng = random.Random(n)
    vals = orc.gt_pow_many(base, _rs(rng, n))
    sc = _rs(rng, n)
    sc[0] = [0, 1, ops.R - 1, 0xD201000000010000][n % 4]
    ctx = ops.ctx()
    ctx.set_tuning(_lib.TUNE_GT_LANES, teams)
    try:
        got = ops.split(ops.gt_pow(b"".join(vals), sc), 576)
    finally:
        ctx.set_tuning(_lib.TUNE_GT_LANES, 0)
    assert got == [orc.gt_pow_many(v, [s])[0] for v, s in zip(vals, sc)]
    assert ops.split(ops.fp12_mul(b"".join(vals), b"".join(got)), 576) == [orc.fp12_mul(a, b) for a, b in zip(vals, got)]


@pytest.mark.parametrize("n,count", [(2, 1), (2, 7), (4, 1), (8, 3), (16, 4), (16, 5), (32, 6), (64, 1), (16, 31)])
def test_transforms(base, n, count):
    """Warp-uniform twiddles (blocks x arrays >= 5, padded to fives) and mixed ones."""
    rng = random.Random(n * 100 + count)
    vals = orc.gt_pow_many(base, _rs(rng, n * count))
    for inv in (False, True):
        got = ops.split(ops.gt_ntt_many(b"".join(vals), n, inverse=inv), 576)
        for q in range(count):
            assert got[n * q : n * (q + 1)] == orc.gt_ntt(vals[n * q : n * (q + 1)], inverse=inv)


@pytest.mark.parametrize("n,keep", [(2, 1), (8, 1), (8, 3), (16, 5), (16, 8), (32, 11)])
def test_prefix_of_any_length(base, n, keep):
    """Of GT values the outputs are canonical: equal to the whole transform's."""
    rng = random.Random(n + keep)
    vals = orc.gt_pow_many(base, _rs(rng, n))
    assert ops.split(ops.cyclotomic_prefix_ifft(b"".join(vals), keep), 576) == orc.gt_ntt(vals, inverse=True)[:keep]


@pytest.mark.parametrize("n", [1, 4, 5, 6, 11])
def test_miller_loops_and_final_exponentiation(n):
    rng = random.Random(40 + n)
    p = orc.g1_mul_many(orc.g1_generator(), _rs(rng, n))
    q = orc.g2_mul_many(orc.g2_generator(), _rs(rng, n))
    if n > 4:
        p[2], q[3] = bytes(96), bytes(192)
    P, Q = b"".join(p), b"".join(q)
    expect = [orc.pairing(a, b) for a, b in zip(p, q)]
    f = ops.miller_loop(P, Q)
    assert ops.split(ops.final_exp(f), 576) == expect
    g = ops.miller_loop_lines(ops.prepare_lines(Q), P)
    assert ops.split(ops.final_exp(ops.final_exp(g, mode=1), mode=2), 576) == expect
    whole = ops.final_exp(ops.multi_miller_loop(P, Q, [0, 0, n // 2, n]))
    parts = []
    for lo, hi in ((0, 0), (0, n // 2), (n // 2, n)):
        acc = orc.fp12_one()
        for e in expect[lo:hi]:
            acc = orc.fp12_mul(acc, e)
        parts.append(acc)
    assert ops.split(whole, 576) == parts


def test_zero_has_no_easy_part():
    f = ops.miller_loop(orc.g1_generator(), orc.g2_generator())
    got = ops.split(ops.final_exp(f + bytes(576) + f, mode=1), 576)
    assert got[1] == bytes(576) and got[0] == got[2]
