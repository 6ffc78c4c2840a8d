"""The reference-named chunk entry point on the tensor path (f32 activations as three bf16 planes) against the layer in
float64, at the edges of its 128-token x 256-output tiles and of its split contractions."""
import ctypes as C

import numpy as np
import pytest

from cwick_b200 import lib as cl, synth
from cwick_b200.compat import Err, make_spec, tensor, tensor_fp8

pytestmark = pytest.mark.gpu


def _layer(x, w, rows0, eps, nh, nope, vdim):
    """(outputs, new cache rows) of the latent layer in float64; the cached rows and the absorbed query as bf16."""
    def bf(a):
        return synth.bf16_to_f32(synth.f32_to_bf16(np.asarray(a, np.float32))).astype(np.float64)

    def norm(a):
        return a / np.sqrt((a * a).mean(-1, keepdims=True) + eps)
    qa, qb, kva, kvb, o = (synth.bf16_to_f32(t).astype(np.float64) for t in w)
    q = (norm(x @ qa.T) @ qb.T).reshape(len(x), nh, nope)
    new = norm(x @ kva.T)
    stored = (new.astype(np.float32).view(np.uint32) & np.uint32(0xFFFF0000)).view(np.float32)      # (the cache-row write truncates)
    lat = np.concatenate([rows0, stored.astype(np.float64)])
    kvb = kvb.reshape(nh, nope + vdim, -1)
    qabs = bf(np.einsum("thr,hrc->thc", q, kvb[:, :nope]))
    s = np.einsum("thc,kc->thk", qabs, lat) / np.sqrt(nope)
    s[np.broadcast_to(np.arange(len(lat)) > (len(rows0) + np.arange(len(x)))[:, None, None], s.shape)] = -np.inf
    p = np.exp(s - s.max(-1, keepdims=True))
    c = bf(np.einsum("thk,kc->thc", p / p.sum(-1, keepdims=True), lat))
    return np.einsum("thc,hrc->thr", c, kvb[:, nope:]).reshape(len(x), -1) @ o.T, new


@pytest.mark.parametrize("bf16_cache", [True, False])
@pytest.mark.parametrize("n,pos0", [(4, 0), (127, 1), (128, 0), (129, 70), (300, 0)])
@pytest.mark.parametrize("H,nh,nope,vdim,q_lora,kv_lora", [(320, 4, 64, 80, 192, 128), (1024, 64, 128, 128, 576, 512)])
def test_chunk_against_the_layer_in_double(monkeypatch, H, nh, nope, vdim, q_lora, kv_lora, n, pos0, bf16_cache):
    monkeypatch.setenv("CWICK_LATENT_BF16", "1" if bf16_cache else "0")
    L = cl.load()
    fn = L["cwick_attention_mla_prefill_chunk"]
    fn.restype = C.c_int
    fn.argtypes = [C.c_void_p] * 10 + [C.c_int64] * 4 + [C.c_void_p] * 5
    L.cwk_dropin_reset()
    shapes = [(q_lora, H), (nh * nope, q_lora), (kv_lora, H), (nh * (nope + vdim), kv_lora), (H, nh * vdim)]
    w = [synth.normal_bf16(5, i, s, s[1] ** -0.5) for i, s in enumerate(shapes)]
    ones = synth.f32_to_bf16(np.ones(max(q_lora, kv_lora), np.float32))
    t = [tensor(a, *s) for a, s in zip(w, shapes)] + [tensor(ones, 1, q_lora), tensor(ones, 1, kv_lora)]
    spec = make_spec(H, nh, nope, vdim, q_lora, kv_lora, 1e-6)
    x = synth.normal(5, 11, n * H).reshape(n, H).astype(np.float32)
    prefix = synth.normal_bf16(5, 12, (pos0 + n, kv_lora))
    cache = prefix.copy() if bf16_cache else synth.bf16_to_f32(prefix)
    out, err = np.zeros((n, H), np.float32), Err()
    st = fn(C.addressof(spec), *[C.byref(a) for a in t], cache.ctypes.data, None, pos0 + n, pos0, n, 0, None, None, x.ctypes.data,
            out.ctypes.data, C.byref(err))
    assert st == 0 and err.status == 0, err.message
    want, rows = _layer(x.astype(np.float64), w, synth.bf16_to_f32(prefix[:pos0]).astype(np.float64), 1e-6, nh, nope, vdim)
    got_rows = synth.bf16_to_f32(cache[pos0:]) if bf16_cache else cache[pos0:]
    np.testing.assert_allclose(got_rows, rows, atol=2e-5 * np.abs(rows).max(), rtol=8e-3 if bf16_cache else 2e-5)
    assert np.linalg.norm(out - want) < 6e-3 * np.linalg.norm(want)
    assert np.array_equal(cache[:pos0], prefix[:pos0] if bf16_cache else synth.bf16_to_f32(prefix[:pos0]))
    L.cwk_dropin_reset()


@pytest.mark.parametrize("n,pos0", [(4, 0), (5, 1), (35, 70), (300, 0)])
@pytest.mark.parametrize("H,nh,nope,vdim,q_lora,kv_lora", [(512, 4, 96, 128, 256, 512),      # a head width that is no multiple of 64
                                                           (264, 3, 40, 72, 512, 256)])      # and contractions that are no multiples of 256
def test_chunk_off_the_tensor_path(monkeypatch, H, nh, nope, vdim, q_lora, kv_lora, n, pos0):
    """Layers that the tensor path refuses: row kernels over groups of four tokens and rows, with remainders of both."""
    test_chunk_against_the_layer_in_double(monkeypatch, H, nh, nope, vdim, q_lora, kv_lora, n, pos0, True)


@pytest.mark.parametrize("pos", [0, 1, 257, 2000])
@pytest.mark.parametrize("kind", ["bf16", "f32", "fp8"])
@pytest.mark.parametrize("H,nh,q_lora", [(1024, 64, 640), (336, 2, 208), (48, 1, 16)])
def test_token_against_the_layer_in_double(monkeypatch, H, nh, q_lora, kind, pos):
    """One-token decode at latent 512 and value heads of 128: rows per block even and odd, fewer rows than blocks, activations
    shorter than a warp's reads, one split record and many."""
    import torch
    nope = vdim = 128
    kv_lora = 512
    monkeypatch.setenv("CWICK_LATENT_BF16", "1")
    L = cl.load()
    fn = L["cwick_attention_mla_decode"]
    fn.restype = None
    fn.argtypes = [C.c_void_p] * 11 + [C.c_int64] * 3 + [C.c_void_p] * 5
    L.cwk_dropin_reset()
    shapes = [(q_lora, H), (nh * nope, q_lora), (kv_lora, H), (nh * (nope + vdim), kv_lora), (H, nh * vdim)]
    w = [synth.normal_bf16(6, i, s, s[1] ** -0.5) for i, s in enumerate(shapes)]
    keep, t, wide = [], [], []
    for i, (a, s) in enumerate(zip(w, shapes)):
        if kind == "f32" and i != 3:
            b = synth.bf16_to_f32(a)
            t.append(tensor(b, *s))
            t[-1].kind = 2
            keep.append(b)
        elif kind == "fp8" and i != 3:
            c = (torch.from_numpy(synth.bf16_to_f32(a)) * 16).to(torch.float8_e4m3fn)
            b, sc = c.view(torch.uint8).numpy(), np.full(((s[0] + 127) // 128, (s[1] + 127) // 128), 1 / 16, np.float32)
            sc[-1, -1] = 1 / 32
            t.append(tensor_fp8(b, sc, *s))
            keep += [b, sc]
            a = synth.f32_to_bf16((c.float().numpy() * np.repeat(np.repeat(sc, 128, 0), 128, 1)[:s[0], :s[1]]).astype(np.float32))
        else:
            t.append(tensor(a, *s))
        wide.append(a)
    ones = synth.f32_to_bf16(np.ones(max(q_lora, kv_lora), np.float32))
    t += [tensor(ones, 1, q_lora), tensor(ones, 1, kv_lora)]
    spec = make_spec(H, nh, nope, vdim, q_lora, kv_lora, 1e-6)
    x = synth.normal(6, 11, H).astype(np.float32)
    cache = synth.normal_bf16(6, 12, (pos + 1, kv_lora))
    before = cache[:pos].copy()
    out, err = np.zeros(H, np.float32), Err()
    ref = C.byref
    fn(C.addressof(spec), ref(t[0]), ref(t[1]), ref(t[2]), ref(t[3]), None, ref(t[4]), ref(t[5]), ref(t[6]), cache.ctypes.data, None, pos + 1, pos, 0,
       None, None, x.ctypes.data, out.ctypes.data, ref(err))
    assert err.status == 0, err.message
    want, rows = _layer(x[None].astype(np.float64), wide, synth.bf16_to_f32(before).astype(np.float64), 1e-6, nh, nope, vdim)
    np.testing.assert_allclose(synth.bf16_to_f32(cache[pos:]), rows, atol=2e-5 * np.abs(rows).max(), rtol=8e-3)
    assert np.linalg.norm(out - want[0]) < 8e-3 * np.linalg.norm(want)
    assert np.array_equal(cache[:pos], before)
    L.cwk_dropin_reset()
