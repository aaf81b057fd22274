"""Scratch of the launchers that cannot be had: nothing is launched on it, nothing
stays allocated, and the caller is told."""
import ctypes

import pytest

from host_runtime import i64, library, log

WBTE_ERR_OOM = -3


@pytest.mark.parametrize("fail_at", [0, 1, 2])
def test_runs_of_prepared_miller_loops(fail_at):
    h = library()
    h.fake_log()
    before = h.fake_live()
    h.fake_fail_at(fail_at)
    ok = h.h_miller_lines_multi(*i64(100, 100, 3))
    h.fake_fail_at(0)
    launches, _ = log(h)
    assert h.fake_live() == before
    assert bool(ok) == (fail_at == 0) and (len(launches) == 3) == (fail_at == 0)
    assert (h.fake_error() != 0) == (fail_at != 0)


@pytest.mark.parametrize("scheme", ["wbtx", "wpfe"])
def test_a_call_without_memory_says_so(scheme):
    """Whichever of a call's allocations fails, its own or a launcher's."""
    h = library()
    ctx = ctypes.c_void_p()
    assert h.wbte_ctx_create(0, ctypes.c_uint64(0), ctypes.byref(ctx)) == 0
    u = ctypes.c_uint64
    B, T, K = 8, 3, 1
    buf = h.fake_buffer(u(1 << 30))
    p = ctypes.c_void_p(buf)

    def call():
        if scheme == "wbtx":
            return h.wbte_wbtx_decrypt_many(ctx, p, p, p, p, p, p, p, p, u(T), u(B), u(K))
        return h.wbte_wpfe_open_many(ctx, p, p, u(T), p, p, p, p, p, p, p, p, u(B), u(K))

    assert call() == 0  # the twiddles of a context stay
    before, count = h.fake_live(), h.fake_allocations()
    assert call() == 0
    count = h.fake_allocations() - count
    assert h.fake_live() == before and count > 5
    for k in range(1, count + 1):
        h.fake_fail_at(k)
        code = call()
        h.fake_fail_at(0)
        assert (k, code) == (k, WBTE_ERR_OOM)
        assert h.fake_live() == before
    h.wbte_ctx_destroy(ctx)
    h.fake_free(p)
