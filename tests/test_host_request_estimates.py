"""The memory that requests are admitted by, against what the calls of a request
allocate."""
import ctypes

import pytest

from host_runtime import library
from weighted_bte_b200 import _lib, serving, wpfe_batched
from weighted_bte_b200 import weighted_btx as wb

WBTE_ERR_OOM = -3
G1B, G2B, GTB, LINES = 96, 192, 576, 68 * 288
u = ctypes.c_uint64
SHAPES = [(1, 1), (8, 3), (32, 24), (128, 24), (512, 3), (512, 9), (2048, 1), (2048, 3), (2048, 24), (8192, 9)]


@pytest.fixture
def run():
    """run(name, args..) -> the bytes that a call of the C interface allocates at once."""
    h = library()
    ctx = ctypes.c_void_p()
    assert h.wbte_ctx_create(0, u(0), ctypes.byref(ctx)) == 0
    buf = ctypes.c_void_p(h.fake_buffer(u(1 << 34)))

    def peak(name, *args):
        call = lambda: getattr(h, name)(ctx, *(buf if a is None else a for a in args))  # noqa: E731
        assert call() == 0  # the twiddles of a context stay
        before = h.fake_live()
        h.fake_peak()
        assert call() == 0
        return h.fake_peak() - before

    yield peak
    h.fake_free(buf)
    h.wbte_ctx_destroy(ctx)


def _decrypt(run, scheme, B, T, K, own):
    """own: a host array for the inputs and outputs that the call itself uploads."""
    x = own if own is not None else None
    if scheme == "wbtx":
        return run("wbte_wbtx_decrypt_many", x, None, None, None, x, x, x, x, u(T), u(B), u(K))
    return run("wbte_wpfe_decrypt_many", x, x, u(T), None, None, None, None, x, x, None, u(B), u(K))


@pytest.mark.parametrize("B,T", SHAPES)
def test_weighted_btx(run, B, T):
    need = serving.request_bytes(B, T)
    batch = B * (G1B + GTB + G1B + 32 + 1)
    shared = B * (G1B + GTB + 1) + B * GTB  # a group's arrays and its output
    assert batch + B * GTB + run("wbte_wbtx_precompute", None, None, None, None, u(B)) <= need
    assert batch + 2 * B * GTB + run("wbte_wbtx_open", None, None, None, u(T), None, None, None, u(B)) <= need
    for K in (1, 4, 16):
        assert K * (batch + shared) + _decrypt(run, "wbtx", B, T, K, None) <= K * need


@pytest.mark.parametrize("B,T", SHAPES)
def test_weighted_pfe(run, B, T):
    need = wpfe_batched.request_bytes(B, T)
    for K in (1, 4, 16):
        own = ctypes.create_string_buffer((G1B + 2 * GTB) * B * K + G1B * T * K)
        assert _decrypt(run, "wpfe", B, T, K, own) <= K * need


@pytest.mark.parametrize("scheme", ["wbtx", "wpfe"])
@pytest.mark.parametrize("B,T", SHAPES)
def test_the_native_server_refuses_what_does_not_fit(run, scheme, B, T):
    h = library()
    own = ctypes.create_string_buffer((G1B + 2 * GTB) * B + G1B * T)
    offsets = (ctypes.c_int64 * (T + 1))(*range(T + 1))
    crs, ctx, srv, ticket = ctypes.c_void_p(), ctypes.c_void_p(), ctypes.c_void_p(), u()
    assert h.wbte_ctx_create(0, u(0), ctypes.byref(ctx)) == 0
    key = (_lib.WbtxKey if scheme == "wbtx" else _lib.WpfeKey)()
    for field in key._fields_:
        if field[1] is ctypes.c_void_p:
            setattr(key, field[0], ctypes.addressof(own))
    key.party_offsets = ctypes.addressof(offsets)
    key.party_count = key.total_weight = T
    if scheme == "wbtx":
        key.max_batch_size = B
        assert h.wbte_crs_upload_wbtx(ctx, ctypes.byref(key), ctypes.byref(crs)) == 0
        committee = LINES * wb.transform_size_for(B) + B * T * (G2B + LINES)
    else:
        key.batch_size = B
        assert h.wbte_crs_upload_wpfe(ctx, ctypes.byref(key), own, ctypes.byref(crs)) == 0
        committee = B * T * (G2B + LINES) + 2 * B * LINES
    least = committee + _decrypt(run, scheme, B, T, 1, own)
    assert h.wbte_server_create(0, 1, 1, u(least - 1), ctypes.byref(srv)) == 0
    req = _lib.Request()
    req.crs, req.batch_size, req.party_count = crs, B, T
    req.first = req.second = req.valid = req.sigma = req.messages = ctypes.addressof(own)
    req.party_indices = ctypes.addressof(offsets)
    assert h.wbte_submit(srv, ctypes.byref(req), ctypes.byref(ticket)) == WBTE_ERR_OOM
    h.wbte_server_destroy(srv)
    h.wbte_crs_destroy(crs)
    h.wbte_ctx_destroy(ctx)
