"""What is timed: the calls that a user of the framework makes, over the range of sizes that they are made at.

Each case names a kind of call and its sizes.  The sizes are those of the
repository's configurations (btx with B = 32, N = 16, t = 8; weighted_btx
with B = 512, n = 128 Zipf(1) weights, W = 4096; weighted_pfe batches of
log-uniform sizes under n = 64, W = 2048; MSMs of 2^10 to 2^20 points and
multi-pairings of 1 to 4096 pairs) and ragged sizes in between.

All outputs are bytes (canonical encodings of group elements, digests, masks,
scalars): they are equal or they are wrong, so there is no exact().
"""
from __future__ import annotations

import random

import numpy as np
import torch

from weighted_bte_b200 import btx, ops, pfe, serving, wpfe_batched
from weighted_bte_b200 import weighted_btx as wb
from weighted_bte_b200 import weighted_pfe as wp
from weighted_bte_b200.rng import ChaCha20Rng
from weighted_bte_b200.workloads import minimal_authorized_parties, zipf_weights

G1B, G2B, GTB = 96, 192, 576


def listed():
    return [
        # one small batch through a whole unweighted scheme: latency, many short launches
        {"name": "btx_decrypt_b32", "kind": "btx", "B": 32, "n": 16, "t": 8},
        # the same for partial-fraction encryption at an ordinary size
        {"name": "pfe_decrypt_b128", "kind": "pfe", "B": 128, "n": 16, "t": 8},
        # a served request of odd size, host objects in and out, its committee already prepared
        {"name": "wbtx_request_b100", "kind": "wbtx_request", "B": 100, "n": 64, "W": 2048},
        # a sender's batch: the encode direction
        {"name": "wbtx_encrypt_512", "kind": "wbtx_encrypt", "B": 512, "n": 16, "W": 64},
        # arrival of a batch: encodings, challenges, proof checks, digest
        {"name": "wbtx_validate_512", "kind": "wbtx_validate", "B": 512, "n": 16, "W": 64},
        # the ciphertext-dependent work before the shares arrive, one batch
        {"name": "wbtx_precompute_512", "kind": "wbtx_precompute", "B": 512, "n": 16, "W": 64},
        # a committee that was not seen before, at the benchmark's size: G2 MSMs, G2 transform, line tables
        {"name": "wbtx_prepare_512", "kind": "wbtx_prepare", "B": 512, "n": 128, "W": 4096},
        # the batched form at the benchmark's size: the largest call
        {"name": "wbtx_group_64x512", "kind": "wbtx_group", "B": 512, "K": 64, "n": 128, "W": 4096},
        # uneven weighted_pfe batches in size classes, several streams and threads, padding
        {"name": "wpfe_uneven_24", "kind": "wpfe_uneven", "count": 24, "lo": 8, "hi": 512, "n": 64, "W": 2048},
        # the primitives that other protocols call: MSMs and products of pairings
        {"name": "g1_msm_65536", "kind": "g1_msm", "points": 65536},
        {"name": "g2_msm_20011", "kind": "g2_msm", "points": 20011},
        {"name": "pairing_products_1500", "kind": "pairings", "pairs": 1500, "products": 97},
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["btx", "pfe", "wbtx_request", "wbtx_encrypt", "wbtx_validate", "wbtx_precompute",
                       "wbtx_prepare", "wbtx_group", "wpfe_uneven", "g1_msm", "g2_msm", "pairings"])
    if kind == "btx":
        n = rng.randint(4, 24)
        return {"kind": kind, "B": _log_int(rng, 3, 200), "n": n, "t": rng.randint(1, n - 1)}
    if kind == "pfe":
        n = rng.randint(4, 24)
        return {"kind": kind, "B": 2 ** rng.randint(2, 8), "n": n, "t": rng.randint(1, n - 1)}
    if kind in ("g1_msm", "g2_msm"):
        return {"kind": kind, "points": _log_int(rng, 700, 150000 if kind == "g1_msm" else 60000)}
    if kind == "pairings":
        pairs = _log_int(rng, 8, 4096)
        return {"kind": kind, "pairs": pairs, "products": _log_int(rng, 1, pairs)}
    if kind == "wpfe_uneven":
        n = rng.randint(8, 64)
        return {"kind": kind, "count": rng.randint(3, 40), "lo": rng.randint(4, 16), "hi": _log_int(rng, 40, 256),
                "n": n, "W": n * rng.randint(2, 32)}
    n = rng.randint(6, 128)
    if kind == "wbtx_group":
        B = _log_int(rng, 12, 512)
        most = max(2, min(64, 16384 // B))
        return {"kind": kind, "B": B, "K": _log_int(rng, 2, most), "n": n, "W": n * rng.randint(2, 16)}
    return {"kind": kind, "B": _log_int(rng, 6, 512), "n": n, "W": n * rng.randint(2, 16)}


# ------------------------------------------------------------------ inputs
def _scalars(rng, n):
    return [rng.getrandbits(380) % ops.R for _ in range(n)]


def _messages(rng, n):
    return wb.messages_from_bytes([rng.getrandbits(256).to_bytes(32, "little") for _ in range(n)])


def _sizes(case):
    """The batch sizes of a case, log-uniform; they are the case's, not the seed's."""
    rng = random.Random("sizes %d %d %d" % (case["count"], case["lo"], case["hi"]))
    return [_log_int(rng, case["lo"], case["hi"]) for _ in range(case["count"])]


class _Wbtx:
    """A weighted_btx setup: keys, the heaviest-first committee, a batch."""

    def __init__(self, case, rng, batches=1):
        weights = zipf_weights(case["n"], case["W"])
        t = case["W"] // 3
        self.chacha = ChaCha20Rng.seed_from_u64(rng.getrandbits(63))
        mat = wb.keygen_with_rng(wb.KeygenConfig(case["B"], weights, t), self.chacha)
        self.ek, self.dk = mat.encryption_key, mat.decryption_key
        committee, _ = minimal_authorized_parties(weights, t)
        self.keys = [mat.party_keys[j] for j in committee]
        self.messages = [_messages(rng, case["B"]) for _ in range(batches)]

    def encrypt(self):
        flat = [m for ms in self.messages for m in ms]
        cts = wb.encrypt_many(self.ek, flat, self.chacha)
        B = len(self.messages[0])
        return [cts[B * k : B * (k + 1)] for k in range(len(self.messages))]

    def accept(self, cts):
        batch = wb.validate_batch(self.dk, cts)
        shares = wb.partial_decrypt_many(self.keys, batch)
        return batch, wb.accept_decryption_shares(self.dk, batch, shares, self.chacha)


def prepare(case, seed):
    kind = case["kind"]
    rng = random.Random("%d %s" % (seed, kind))
    state = {"kind": kind, "case": case}
    if kind == "btx":
        chacha = ChaCha20Rng.seed_from_u64(rng.getrandbits(63))
        mat = btx.keygen_with_rng(btx.KeygenConfig(case["B"], case["n"], case["t"]), chacha)
        state["dk"] = mat.decryption_key
        state["servers"] = mat.server_keys[: case["t"] + 1]
        state["cts"] = btx.encrypt_many(mat.encryption_key, _messages(rng, case["B"]), chacha)
        state["kernel"] = btx.MiddleProductKernel(mat.decryption_key, case["B"])
    elif kind == "pfe":
        chacha = ChaCha20Rng.seed_from_u64(rng.getrandbits(63))
        mat = pfe.keygen_with_rng(pfe.KeygenConfig(case["B"], case["n"], case["t"]), chacha)
        state["ek"], state["dk"] = mat.encryption_key, mat.decryption_key
        state["servers"] = mat.server_keys[: case["t"] + 1]
        state["cts"] = pfe.encrypt_many(mat.encryption_key, _messages(rng, case["B"]), chacha)
        state["kernel"] = pfe.PartialFractionKernel(mat.decryption_key)
    elif kind == "wbtx_request":
        s = _Wbtx(case, rng)
        cts = s.encrypt()[0]
        cache = serving.CommitteeCache(8 << 30)
        cache.get(s.dk, s.accept(cts)[1])  # a server holds its committees prepared
        state.update(dk=s.dk, keys=s.keys, cts=cts, cache=cache, chacha=s.chacha)
    elif kind == "wbtx_encrypt":
        s = _Wbtx(case, rng)
        state.update(ek=s.ek, messages=s.messages[0], seed=rng.getrandbits(63))
    elif kind == "wbtx_validate":
        s = _Wbtx(case, rng)
        cts = s.encrypt()[0]
        bad = cts[len(cts) // 2]  # one broken proof
        cts[len(cts) // 2] = wb.Ciphertext(bad.first, bad.second,
                                           wb.SchnorrProof(bad.proof.commitment, (bad.proof.response + 1) % ops.R))
        state.update(dk=s.dk, cts=cts)
    elif kind == "wbtx_precompute":
        s = _Wbtx(case, rng)
        batch, accepted = s.accept(s.encrypt()[0])
        state.update(batch=batch, pre=wb.prepare_decryption(s.dk, accepted))
    elif kind == "wbtx_prepare":
        s = _Wbtx(case, rng)
        state.update(dk=s.dk, accepted=s.accept(s.encrypt()[0])[1])
    elif kind == "wbtx_group":
        s = _Wbtx(case, rng, case["K"])
        batches = s.encrypt()
        cache = serving.CommitteeCache(8 << 30)
        cache.get(s.dk, s.accept(batches[0])[1])
        cache.vk_tables(s.dk, case["B"], [k.party_index for k in s.keys])
        state.update(dk=s.dk, keys=s.keys, cache=cache, chacha=s.chacha,
                     batches=[wb.CiphertextBatch.upload(cts) for cts in batches])
    elif kind == "wpfe_uneven":
        weights = zipf_weights(case["n"], case["W"])
        t = case["W"] // 3
        committee, _ = minimal_authorized_parties(weights, t)
        sizes = _sizes(case)
        classes = wpfe_batched.class_keys([wpfe_batched.size_class(s) for s in sizes], weights, t, committee,
                                          rng.getrandbits(40))
        chacha = ChaCha20Rng.seed_from_u64(rng.getrandbits(63))
        state["batches"] = [wp.encrypt_many(classes[wpfe_batched.size_class(s)].material.encryption_key,
                                            _messages(rng, s), chacha) for s in sizes]
        state["decryptor"] = wpfe_batched.UnevenBatchDecryptor(classes, streams=4)
        smallest = {wpfe_batched.size_class(len(b)): b for b in state["batches"]}
        state["decryptor"].decrypt(list(smallest.values()))  # a server holds its committees prepared
    elif kind in ("g1_msm", "g2_msm"):
        n = case["points"]
        size, mul = (G1B, ops.g1_mul_generator) if kind == "g1_msm" else (G2B, ops.g2_mul_generator)
        state["points"] = torch.empty(size * n, dtype=torch.uint8, device="cuda")
        mul(_scalars(rng, n), out=state["points"])
        state["scalars"] = ops.scalars_bytes(_scalars(rng, n))
        state["out"] = torch.empty(size, dtype=torch.uint8, device="cuda")
    elif kind == "pairings":
        n, k = case["pairs"], case["products"]
        state["p"] = torch.empty(G1B * n, dtype=torch.uint8, device="cuda")
        state["q"] = torch.empty(G2B * n, dtype=torch.uint8, device="cuda")
        ops.g1_mul_generator(_scalars(rng, n), out=state["p"])
        ops.g2_mul_generator(_scalars(rng, n), out=state["q"])
        state["offsets"] = [0] + sorted(rng.sample(range(1, n), k - 1)) + [n]
    else:
        raise ValueError(kind)
    return state


# ------------------------------------------------------------------ the call
def _bytes(*parts):
    return torch.from_numpy(np.frombuffer(b"".join(parts), dtype=np.uint8).copy())


def run(state):
    kind = state["kind"]
    if kind == "btx":
        return _bytes(*btx.decrypt(state["dk"], state["cts"], state["servers"], state["kernel"]))
    if kind == "pfe":
        return _bytes(*pfe.decrypt(state["ek"], state["dk"], state["cts"], state["servers"], state["kernel"]))
    if kind == "wbtx_request":
        return _bytes(*serving.decrypt_request(state["dk"], state["cts"], state["keys"], state["chacha"],
                                               state["cache"]))
    if kind == "wbtx_encrypt":
        cts = wb.encrypt_many(state["ek"], state["messages"], ChaCha20Rng.seed_from_u64(state["seed"]))
        return {"first": _bytes(*(c.first for c in cts)), "second": _bytes(*(c.second for c in cts)),
                "commitment": _bytes(*(c.proof.commitment for c in cts)),
                "response": _bytes(*(c.proof.response.to_bytes(32, "little") for c in cts))}
    if kind == "wbtx_validate":
        v = wb.validate_batch(state["dk"], state["cts"])
        return {"digest": _bytes(v.digest()), "valid": v.valid, "first": v.first_dev}
    if kind == "wbtx_precompute":
        return wb.precompute_batch(state["pre"], state["batch"]).beta
    if kind == "wbtx_prepare":
        pre = wb.prepare_decryption(state["dk"], state["accepted"])
        return {"opening_keys": pre.opening_keys, "opening_lines": pre.opening_lines,
                "kernel": pre.transformed_kernel, "kernel_lines": pre.kernel_lines}
    if kind == "wbtx_group":
        # a batch as it arrives carries no encodings or digest yet
        batches = [wb.CiphertextBatch(b.first, b.second, b.commitment, b.responses) for b in state["batches"]]
        out = serving.decrypt_group(state["dk"], batches, state["keys"], state["chacha"], state["cache"],
                                    device_output=True)
        return torch.stack(out)
    if kind == "wpfe_uneven":
        out = state["decryptor"].decrypt(state["batches"], seed=1)
        return _bytes(*(m for batch in out for m in batch))
    if kind == "g1_msm":
        return ops.g1_msm(state["points"], state["scalars"], out=state["out"])
    if kind == "g2_msm":
        return ops.g2_msm(state["points"], state["scalars"], out=state["out"])
    return _bytes(ops.final_exp(ops.multi_miller_loop(state["p"], state["q"], state["offsets"])))


# ------------------------------------------------------------------ its work
# Fp products: a Miller loop with prepared lines, one that computes its lines,
# the final exponentiation's two parts, a power in GT, a multiple in G1 and G2,
# a mixed addition in G1 and G2.
LINES, LOOP, EASY, HARD, GT_POW, G1_MUL, G2_MUL, G1_ADD, G2_ADD = 5156, 6700, 700, 7497, 4200, 1500, 3200, 10, 28
PRODUCT = 600  # 300 multiply-adds of 32-bit words


def _log2(n):
    return max(1, (n - 1).bit_length())


def _decrypt_products(B, T):
    """validate, partial decryptions, share check, cross terms, opening of one batch."""
    m = 1 << (2 * B - 1).bit_length()
    transform = 3 * (m // 4) * (_log2(m) // 2)
    return (B * (2 * G1_MUL) + T * B * 50 * G1_ADD + B * LOOP + HARD + transform * (G1_MUL + GT_POW)
            + m * (LINES + EASY) + B * (2232 + 2924 * T + EASY + HARD))


def work(case):
    kind = case["kind"]
    if kind in ("g1_msm", "g2_msm"):
        n, size, add = case["points"], *((G1B, G1_ADD) if kind == "g1_msm" else (G2B, G2_ADD))
        return {"bytes": n * (size + 32) + size, "flops": n * (255.0 / _log2(n)) * add * PRODUCT}
    if kind == "pairings":
        n, k = case["pairs"], case["products"]
        return {"bytes": n * (G1B + G2B) + k * GTB, "flops": (n * 4500 + k * (2232 + EASY + HARD)) * PRODUCT}
    record = G1B + GTB + G1B + 32
    if kind in ("btx", "pfe"):
        B = case["B"]
        return {"bytes": B * (record + GTB), "flops": _decrypt_products(B, 1) * PRODUCT}
    if kind == "wpfe_uneven":
        sizes = _sizes(case)
        T = len(minimal_authorized_parties(zipf_weights(case["n"], case["W"]), case["W"] // 3)[0])
        return {"bytes": sum(sizes) * (record + GTB),
                "flops": sum(_decrypt_products(1 << _log2(b), T) for b in sizes) * PRODUCT}
    B, weights = case["B"], zipf_weights(case["n"], case["W"])
    committee, total = minimal_authorized_parties(weights, case["W"] // 3)
    T = len(committee)
    m = 1 << (2 * B - 1).bit_length()
    if kind == "wbtx_encrypt":
        return {"bytes": B * (GTB + record), "flops": B * (2 * G1_MUL + GT_POW) * PRODUCT}
    if kind == "wbtx_validate":
        return {"bytes": B * (record + G1B), "flops": B * 2 * G1_MUL * PRODUCT}
    if kind == "wbtx_precompute":
        transform = 3 * (m // 4) * (_log2(m) // 2)
        return {"bytes": B * G1B + m * 68 * 288 + B * GTB,
                "flops": (transform * (G1_MUL + GT_POW) + m * (LINES + EASY) + B * HARD) * PRODUCT}
    if kind == "wbtx_prepare":
        return {"bytes": 2 * B * total * G2B + (m + B * T) * (G2B + 68 * 288),
                "flops": (2 * B * total * 25 * G2_ADD + m * _log2(m) // 2 * G2_MUL + (m + B * T) * 1500) * PRODUCT}
    K = case.get("K", 1)
    return {"bytes": K * B * (record + GTB) + (m + B * T) * 68 * 288,
            "flops": K * _decrypt_products(B, T) * PRODUCT}
