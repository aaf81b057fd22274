"""Seeded randomness for key generation and encryption.

`ChaCha20Rng` produces the ChaCha20 keystream (RFC 8439 quarter-round and
block function, 20 rounds, 64-bit block counter, zero stream id) as little-
endian 32-bit words; `seed_from_u64` expands a 64-bit seed into the 32-byte
key with the PCG32 sequence that rand_core 0.6's `SeedableRng::seed_from_u64`
publishes.  `random_scalar` draws eight 64-bit words and reduces the 512-bit
little-endian integer modulo r (the wide reduction used by `Scalar::random`
in the ff/bls12_381 family).  `OsRng` mirrors `rand_core::OsRng`.

The reference's tests draw from OsRng only, so these seeded streams are a
convention of this project for reproducible inputs.
"""
from __future__ import annotations

import os
import struct

R = 0x73EDA753299D7D483339D80809A1D80553BDA402FFFE5BFEFFFFFFFF00000001
_M32 = 0xFFFFFFFF
_M64 = 0xFFFFFFFFFFFFFFFF


def _rotl(x: int, n: int) -> int:
    return ((x << n) | (x >> (32 - n))) & _M32


def _quarter(s, a, b, c, d):
    s[a] = (s[a] + s[b]) & _M32
    s[d] = _rotl(s[d] ^ s[a], 16)
    s[c] = (s[c] + s[d]) & _M32
    s[b] = _rotl(s[b] ^ s[c], 12)
    s[a] = (s[a] + s[b]) & _M32
    s[d] = _rotl(s[d] ^ s[a], 8)
    s[c] = (s[c] + s[d]) & _M32
    s[b] = _rotl(s[b] ^ s[c], 7)


def chacha20_block(key_words, counter: int, stream: int = 0):
    state = [0x61707865, 0x3320646E, 0x79622D32, 0x6B206574] + list(key_words) + [
        counter & _M32,
        (counter >> 32) & _M32,
        stream & _M32,
        (stream >> 32) & _M32,
    ]
    w = list(state)
    for _ in range(10):
        _quarter(w, 0, 4, 8, 12)
        _quarter(w, 1, 5, 9, 13)
        _quarter(w, 2, 6, 10, 14)
        _quarter(w, 3, 7, 11, 15)
        _quarter(w, 0, 5, 10, 15)
        _quarter(w, 1, 6, 11, 12)
        _quarter(w, 2, 7, 8, 13)
        _quarter(w, 3, 4, 9, 14)
    return [(w[i] + state[i]) & _M32 for i in range(16)]


def _keystream(key_words, counter: int, n: int) -> bytes:
    """n consecutive keystream blocks (counters counter .. counter + n - 1,
    stream 0).  The four quarter rounds of a column or diagonal round run as one
    on (4, n) arrays of words (the same function as chacha20_block): numpy's
    cost per call, not its arithmetic, bounds blocks by the hundred."""
    import numpy as np

    st = np.empty((16, n), dtype=np.uint32)
    st[0:4] = np.array([0x61707865, 0x3320646E, 0x79622D32, 0x6B206574], dtype=np.uint32)[:, None]
    st[4:12] = np.array(list(key_words), dtype=np.uint32)[:, None]
    ctr = np.arange(counter, counter + n, dtype=np.uint64)
    st[12] = (ctr & np.uint64(_M32)).astype(np.uint32)
    st[13] = (ctr >> np.uint64(32)).astype(np.uint32)
    st[14:16] = 0
    a, b, c, d = (st[4 * i : 4 * i + 4].copy() for i in range(4))
    t = np.empty_like(a)

    def xor_rotl(x, y, k):  # x <- rotl(x ^ y, k)
        np.bitwise_xor(x, y, out=x)
        np.right_shift(x, np.uint32(32 - k), out=t)
        np.left_shift(x, np.uint32(k), out=x)
        np.bitwise_or(x, t, out=x)

    def quarters():
        nonlocal a, c
        a += b
        xor_rotl(d, a, 16)
        c += d
        xor_rotl(b, c, 12)
        a += b
        xor_rotl(d, a, 8)
        c += d
        xor_rotl(b, c, 7)

    for _ in range(10):
        quarters()
        b, c, d = b[[1, 2, 3, 0]], c[[2, 3, 0, 1]], d[[3, 0, 1, 2]]
        quarters()
        b, c, d = b[[3, 0, 1, 2]], c[[2, 3, 0, 1]], d[[1, 2, 3, 0]]
    return (np.concatenate([a, b, c, d]) + st).T.astype("<u4").tobytes()


def chacha20_blocks(key_words, counter: int, n: int):
    """The words of _keystream as one flat list of 16 n integers."""
    return list(struct.unpack(f"<{16 * n}I", _keystream(key_words, counter, n)))


def _pcg32(state: int):
    state = (state * 6364136223846793005 + 11634580027462260723) & _M64
    xorshifted = (((state >> 18) ^ state) >> 27) & _M32
    rot = state >> 59
    x = ((xorshifted >> rot) | (xorshifted << ((32 - rot) & 31))) & _M32
    return state, x


class ChaCha20Rng:
    def __init__(self, seed: bytes):
        if len(seed) != 32:
            raise ValueError("ChaCha20Rng takes a 32-byte seed")
        self.key = list(struct.unpack("<8I", seed))
        self.counter = 0
        self._stream, self._at = b"", 0
        self._refill = 0

    @classmethod
    def seed_from_u64(cls, state: int) -> "ChaCha20Rng":
        words = []
        s = state & _M64
        for _ in range(8):
            s, x = _pcg32(s)
            words.append(x)
        return cls(struct.pack("<8I", *words))

    # keystream blocks of the first refill, doubled up to 16 times that: the
    # words come out in the same order whatever the size (blocks depend only on
    # key and counter)
    REFILL_BLOCKS = 64

    def _take(self, n: int) -> bytes:
        """The next n bytes of the keystream (n a multiple of four)."""
        out = self._stream[self._at : self._at + n]
        self._at += len(out)
        while len(out) < n:
            self._refill = min(max(self.REFILL_BLOCKS, 2 * self._refill), 16 * self.REFILL_BLOCKS)
            self._stream = _keystream(self.key, self.counter, self._refill)
            self.counter += self._refill
            self._at = n - len(out)
            out += self._stream[: self._at]
            self._at = min(self._at, len(self._stream))
        return out

    def next_u32(self) -> int:
        return int.from_bytes(self._take(4), "little")

    def next_u64(self) -> int:
        return int.from_bytes(self._take(8), "little")

    def fill_bytes(self, n: int) -> bytes:
        return self._take((n + 3) // 4 * 4)[:n]


class OsRng:
    def next_u64(self) -> int:
        return int.from_bytes(os.urandom(8), "little")

    def fill_bytes(self, n: int) -> bytes:
        return os.urandom(n)


def random_scalar(rng) -> int:
    """A scalar from eight 64-bit words of `rng`, least significant first.  `rng` is
    anything with next_u64; the generators of this file give the words as the 64
    bytes they are, in one call."""
    if type(rng) in (ChaCha20Rng, OsRng):
        return int.from_bytes(rng.fill_bytes(64), "little") % R
    acc = 0
    for i in range(8):
        acc |= rng.next_u64() << (64 * i)
    return acc % R


def sample_nonzero(rng) -> int:
    while True:
        s = random_scalar(rng)
        if s:
            return s
