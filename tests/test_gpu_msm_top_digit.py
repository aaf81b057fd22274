"""MSMs over scalars of all 256 bits: the highest digit of windows that end at bit
256 has none to carry into."""
import random

import pytest

pytestmark = pytest.mark.gpu

from weighted_bte_b200 import _lib, ops  # noqa: E402


@pytest.mark.parametrize("window", [0, 4, 8, 13])
@pytest.mark.parametrize("n", [5, 33, 700, 20011])
def test_scalars_of_256_bits(n, window):
    rng = random.Random(n)
    u = [rng.randrange(ops.R) for _ in range(101)]
    edge = [(1 << 256) - 1, 1 << 255, (1 << 255) - 1, 0x80 << 248, 0xFF << 248, (0x81 << 248) - 1, ops.R, 0]
    s = (edge + [rng.randrange(1 << 256) for _ in range(n)])[:n]
    sc = b"".join(x.to_bytes(32, "little") for x in s)
    total = sum(a * u[i % len(u)] for i, a in enumerate(s))
    tile = lambda b, size: (b * (n // len(u) + 1))[: size * n]  # noqa: E731
    ctx = ops.ctx()
    ctx.set_tuning(_lib.TUNE_MSM_WINDOW, window)
    try:
        got = [bytes(f(tile(bytes(g(u)), z), sc)) for f, g, z in
               [(ops.g1_msm, ops.g1_mul_generator, 96), (ops.g2_msm, ops.g2_mul_generator, 192)]]
    finally:
        ctx.set_tuning(_lib.TUNE_MSM_WINDOW, 0)
    assert got == [bytes(ops.g1_mul_generator([total])), bytes(ops.g2_mul_generator([total]))]
