"""Scalars drawn from a caller's own generator, which has next_u64 alone."""
from weighted_bte_b200.rng import R, ChaCha20Rng, random_scalar, sample_nonzero


class Words:
    def __init__(self, words):
        self.words = list(words)

    def next_u64(self):
        return self.words.pop(0)


class Complement(ChaCha20Rng):
    def next_u64(self):
        return super().next_u64() ^ ((1 << 64) - 1)


def _scalar(words):
    return sum(w << (64 * i) for i, w in enumerate(words)) % R


def test_a_generator_of_words():
    words = [(0x9E3779B97F4A7C15 * (i + 1)) % (1 << 64) for i in range(8)]
    assert random_scalar(Words(words)) == _scalar(words)
    assert sample_nonzero(Words([0] * 8 + words)) == _scalar(words)


def test_a_generator_that_changes_the_words():
    plain = ChaCha20Rng.seed_from_u64(5)
    words = [plain.next_u64() ^ ((1 << 64) - 1) for _ in range(8)]
    assert random_scalar(Complement.seed_from_u64(5)) == _scalar(words)


def test_the_library_s_own_generators_draw_the_same_words():
    a, b = ChaCha20Rng.seed_from_u64(6), ChaCha20Rng.seed_from_u64(6)
    assert [random_scalar(a) for _ in range(40)] == [_scalar([b.next_u64() for _ in range(8)]) for _ in range(40)]
