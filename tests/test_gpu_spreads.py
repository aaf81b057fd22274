"""How a launch is spread over lanes at sizes between the smallest and the largest:
runs of prepared pairings of every length, with ragged last runs, and fixed-base
sums of one, four and sixteen pairs of lanes an output."""
import random

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from oracle import oracle as orc  # noqa: E402
from weighted_bte_b200 import _lib, ops  # noqa: E402
from weighted_bte_b200 import weighted_btx as wb  # noqa: E402
from weighted_bte_b200.rng import ChaCha20Rng  # noqa: E402


# pairings of a slot and slots of a call: on 148 SMs teams of twelve with runs of
# one and three, teams of six with runs of 1, 2, 3, 4, 5, 7 and 9
@pytest.mark.parametrize("T,n", [(1, 36), (2, 1204), (2, 3000), (3, 900), (3, 2020), (3, 2460), (5, 500), (5, 1300), (5, 1600),
                                 (5, 3700), (5, 4100), (7, 900), (7, 1000), (7, 2300), (7, 4100), (9, 700), (9, 1000),
                                 (9, 2460), (9, 4700)])
def test_openings(T, n):
    rng = random.Random(100 * T + n)
    B, K = 4, n // 4
    a, b = orc.g1_mul_many(orc.g1_generator(), [rng.randrange(ops.R) for _ in range(2)])
    g1 = [a, orc.g1_neg(a), b, bytes(96)]
    g2 = orc.g2_mul_many(orc.g2_generator(), [rng.randrange(ops.R) for _ in range(3)]) + [bytes(192)]
    s = lambda k, t: (k + t * t) % 4  # noqa: E731
    q = lambda i, t: (i + 2 * t) % 4  # noqa: E731
    # alpha is divided out: pairings of the negatives
    pairing = [[orc.pairing(orc.g1_neg(x), y) for y in g2] for x in g1]
    want = {}
    for k in range(4):
        for i in range(B):
            acc = orc.fp12_one()
            for t in range(T):
                acc = orc.fp12_mul(acc, pairing[s(k, t)][q(i, t)])
            want[k, i] = acc
    keys = b"".join(g2[q(i, t)] for i in range(B) for t in range(T))
    sigma = b"".join(g1[s(k, t)] for k in range(K) for t in range(T))
    one = orc.fp12_one() * (B * K)
    out = bytearray(576 * B * K)
    ops.ctx().call("wbte_wbtx_open_many", out, keys, ops.prepare_lines(keys), sigma, T, one, one, b"\x01" * (B * K), B, K)
    assert ops.split(out, 576) == [want[k % 4, i] for k in range(K) for i in range(B)]


@pytest.mark.parametrize("K", [5, 220, 230, 300, 1360, 1500])
def test_share_checks_over_fixed_tables(K):
    """Eight slots a batch and three keys, two of them the same one with challenges
    that may cancel: aggregates that are wrong anywhere fail the check."""
    rng = ChaCha20Rng.seed_from_u64(31)
    mat = wb.keygen_with_rng(wb.KeygenConfig(8, [3, 2, 4, 1], 4), rng)
    dk = mat.decryption_key
    B, parties = 8, [0, 0, 2]
    T, kinds = len(parties), 3
    batches = []
    for _ in range(kinds):
        msgs = wb.messages_from_bytes([rng.fill_bytes(32) for _ in range(B)])
        batches.append(wb.validate_batch(dk, wb.encrypt_many(mat.encryption_key, msgs, rng)))
    import torch

    first = torch.cat([batches[k % kinds].first_dev[: 96 * B] for k in range(K)])
    shares = [b"".join(s.sigma for s in wb.partial_decrypt_many([mat.party_keys[p] for p in parties], b)) for b in batches]
    sig = bytearray(b"".join(shares[k % kinds] for k in range(K)))
    r = random.Random(K)
    c = [r.randrange(ops.R) for _ in range(6)]
    rows = [[c[0], c[1], c[2]], [c[3], ops.R - c[3], c[4]], [c[5], ops.R - c[5], 0], [1, ops.R - 1, 1], [0, 1, 0], [1, 1, 1],
            [ops.R - 1, ops.R - 1, 1 << 200]]
    ch = b"".join(wb.fr_bytes(x) for k in range(K) for x in rows[k % len(rows)])
    bad = sorted({0, K // 2, K - 1})
    want = [1] * K
    for k in bad:
        sig[96 * (k * T + 1) : 96 * (k * T + 2)] = shares[k % kinds][192:288]  # another party's share
        want[k] = 0 if rows[k % len(rows)][1] else 1
    tables = wb.empty_device(_lib.FIXED_TABLE_BYTES * T * B)
    ctx = wb._ctx()
    ctx.call("wbte_wbtx_vk_tables", tables, dk.abi_key(), _lib.i64_array(parties), T, B)
    ok = np.zeros(K, dtype=np.int32)
    ctx.call("wbte_wbtx_verify_shares_many", ok, dk.abi_key(), first, B, bytes(sig), _lib.i64_array(parties), ch, T, K, tables)
    assert list(ok) == want


@pytest.mark.parametrize("n", [1, 7, 1184, 1185])
def test_torus_encodings(n):
    rng = random.Random(n)
    gen = orc.pairing(orc.g1_generator(), orc.g2_generator())
    kinds = orc.gt_pow_many(gen, [rng.randrange(ops.R) for _ in range(6)]) + [orc.fp12_one()]
    tile = lambda v: (v * (n // len(v) + 1))[:n]  # noqa: E731
    assert ops.split(ops.gt_compress(b"".join(tile(kinds)), n), 289) == tile([orc.gt_compress(v) for v in kinds])
