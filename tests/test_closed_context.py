"""Calls on a context that has been closed reach the library with no context, whichever way they are bound, and come back
as an argument error. On the CPU: the context is a stand-in, and what the bound calls are handed is recorded."""
import ctypes as C
from types import SimpleNamespace

import pytest
import torch

from cwick_b200 import lib, ops

FAST = ["cwk_mla_decode", "cwk_gqa_decode", "cwk_dsa_select", "cwk_gdn_scan"]


@pytest.fixture
def attn(monkeypatch):
    def create(device, out):
        C.cast(out, C.POINTER(C.c_void_p))[0] = 0x1000
        return lib.OK
    stub = SimpleNamespace(cwk_ctx_create=create, cwk_ctx_destroy=lambda h: None, cwk_ctx_set_stream=lambda h, s: lib.OK,
                           cwk_last_error=lambda h: b"no context" if h is None else b"")
    handed = []

    def fast(_, name):
        def call(ctx, *args):
            handed.append(ctx)
            return lib.ERR_ARGUMENT if ctx is None else lib.OK
        return call
    monkeypatch.setattr(lib, "load", lambda: stub)
    monkeypatch.setattr(lib, "fast", fast)
    monkeypatch.setattr(ops, "_bf16", lambda t: t)
    monkeypatch.setattr(torch.cuda, "set_device", lambda d: None)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda d: SimpleNamespace(cuda_stream=0))
    a = ops.Attn(0)
    a.handed = handed
    return a


def _call(attn, name):
    def bf(*s):
        return torch.zeros(*s, dtype=torch.bfloat16)

    def f32(*s):
        return torch.zeros(*s)
    one = torch.ones(1, dtype=torch.int32)
    if name == "cwk_mla_decode":
        attn.mla_decode(bf(1, 2, 576), bf(1, 1, 576), one)
    elif name == "cwk_gqa_decode":
        attn.gqa_decode(bf(1, 2, 64), bf(1, 1, 1, 64), bf(1, 1, 1, 64), one)
    elif name == "cwk_dsa_select":
        attn.dsa_select(torch.zeros(1, 1, 128, dtype=torch.uint8), f32(1, 1), f32(1, 1, 128), f32(1, 1), one, 1)
    else:
        attn.gdn_scan(f32(1, 1, 384), f32(1, 1, 1), f32(1, 1, 1), f32(1, 1, 128), f32(1), f32(1), f32(128), f32(1, 1, 128, 128), 1, 1e-6)


@pytest.mark.parametrize("name", FAST)
def test_the_handle_is_read_at_the_call(attn, name):
    _call(attn, name)
    assert attn.handed == [0x1000]
    attn.ctx.close()
    with pytest.raises(lib.CwkError) as e:
        _call(attn, name)
    assert e.value.status == lib.ERR_ARGUMENT and attn.handed == [0x1000, None]


@pytest.mark.parametrize("name", FAST)
@pytest.mark.parametrize("bound", ["compiled", "ctypes"])
def test_the_library_refuses_a_missing_context(name, bound):
    L = lib.load()
    fn = lib.fast(L, name) if bound == "compiled" else getattr(L, name)
    args = [0.0 if a is C.c_float else None if a is C.c_void_p else 1 for a in lib.SIGNATURES[name][1]]
    assert fn(*args) == lib.ERR_ARGUMENT
