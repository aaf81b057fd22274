"""The plan of a Pippenger MSM: the library's own against its restatement for the
product counts, and the fixed-footprint MSM's under its limit."""
import ctypes

import pytest

from host_runtime import library, log
from weighted_bte_b200 import workcount as wc

STATIC_BYTES = (8 << 20) - 256
u = ctypes.c_uint64


def _plan(h, g2, n, k, limit=0):
    out = (ctypes.c_int64 * 3)()
    h.h_msm_plan(2 if g2 else 1, ctypes.c_int64(n), ctypes.c_int64(k), u(limit), out)
    return tuple(out)


@pytest.mark.parametrize("g2", [False, True])
@pytest.mark.parametrize("k", [1, 3, 512])
def test_the_restatement_is_the_library_s(g2, k):
    h = library()
    h.fake_per_sm(4)
    for n in [1, 2, 5, 31, 32, 33, 460, 512, 1382, 4096, 16384, 20011, 65536, 150000, 1 << 20]:
        c, segments, scratch = _plan(h, g2, n, k)
        assert (c, segments) == wc.msm_plan(n, k, g2)
        assert scratch == wc.msm_scratch_bytes(n, k, g2, (256 + c - 1) // c, segments)


def test_plans_of_the_measured_sizes():
    assert wc.msm_plan_window(65536) == 8 and wc.msm_plan_window(1 << 20) == 7


@pytest.mark.parametrize("n", [1, 2, 40, 517, 1000, 3000, 4096, 8191, 12000, 16000, 16383, 16384])
def test_the_fixed_footprint_takes_the_best_plan_that_fits(n):
    h = library()
    buf = ctypes.c_void_p(h.fake_buffer(u(1 << 22)))
    h.fake_per_sm(4)
    c, segments = wc.msm_plan(n, 1, False, limit=STATIC_BYTES)
    h.fake_log()
    assert h.wbte_g1_msm_static(buf, buf, buf, u(n), None) == 0
    (blocks,) = [grid for name, grid, _ in log(h)[0] if "k_segments" in name]
    assert blocks == -(-((256 + c - 1) // c * segments) // 64)
    h.fake_free(buf)


GPUS = [(20, 1), (20, 32), (60, 4), (148, 1), (148, 2), (148, 8), (148, 16), (148, 32), (300, 4), (300, 32)]


@pytest.mark.parametrize("at", range(len(GPUS)))
def test_every_size_of_the_fixed_footprint_runs(at):
    """Whatever a GPU's occupancy makes the plan favour."""
    h = library()
    sms, per_sm = GPUS[at]
    h.fake_device(at + 1, sms)  # waves are kept per device
    h.fake_per_sm(per_sm)
    buf = ctypes.c_void_p(h.fake_buffer(u(1 << 22)))
    try:
        for n in [1, 2, 3, 100, 5000, 10000, 16384]:
            assert h.wbte_g1_msm_static(buf, buf, buf, u(n), None) == 0
            h.fake_log()
    finally:
        h.fake_device(0, 148)
        h.fake_per_sm(4)
        h.fake_free(buf)
