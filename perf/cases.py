"""Performance cases: the attention work of the three model families this engine serves, through its public entry points.

A case names a kind of call and its sizes. Widths are those of the repository's own configurations (latent 512 + rope 64,
64 heads; 16 query / 4 KV heads of 256; 32 Gated DeltaNet heads of 128 x 128; a layer of hidden 4096 for the
reference-named entry points); what varies is what varies in serving: sequences in a batch, tokens cached, tokens in a
prompt, ragged lengths, the weights' data type.
"""
import ctypes as C
import math
import os

import numpy as np
import torch

from cwick_b200 import compat, lib, synth
from cwick_b200.ops import Attn

DEV = "cuda:0"

# MLA layer (hidden, heads, per-head widths, low-rank widths)
HIDDEN, HEADS, NOPE, ROPE, VDIM, Q_LORA, LATENT = 4096, 64, 128, 64, 128, 1536, 512
MLA_SCALE = 1.0 / math.sqrt(NOPE + ROPE)
# lightning indexer
IDX_HEADS, IDX_DIM, IDX_TOPK = 64, 128, 2048
# GQA layer and Gated DeltaNet layer
GQ_HEADS, GQ_KV, GQ_DIM = 16, 4, 256
GDN_HEADS, GDN_DIM, GDN_GROUP = 32, 128, 2
# rows of room behind a sequence that decodes token by token through the reference-named entry point
ENGINE_ROOM, ENGINE_CHUNK = 1024, 512


def listed():
    return [
        # one user's next token, MLA layer with 8192 tokens cached: latency
        {"name": "mla_decode_1x8192", "kind": "mla_decode", "batch": 1, "cached": 8192, "ragged": False},
        # a full serving batch at long contexts, every sequence at its own length: cache bandwidth
        {"name": "mla_decode_64x32768_ragged", "kind": "mla_decode", "batch": 64, "cached": 32768, "ragged": True},
        # sparse decode of long contexts: indexer scores, top 2048, attention over the selected rows
        {"name": "dsa_decode_8x65536", "kind": "dsa_decode", "batch": 8, "cached": 65536, "ragged": False},
        # a whole prompt through an MLA layer with FP8 projections: q/kv projections, attention, un-absorb, o_proj
        {"name": "mla_prompt_4096", "kind": "mla_prompt", "tokens": 4096, "before": 0},
        # the odd-sized last chunk of a longer prompt
        {"name": "mla_prompt_509_after_3001", "kind": "mla_prompt", "tokens": 509, "before": 3001},
        # GQA layer: one user's next token, then an ordinary ragged serving batch
        {"name": "gqa_decode_1x4096", "kind": "gqa_decode", "batch": 1, "cached": 4096, "ragged": False},
        {"name": "gqa_decode_64x4096_ragged", "kind": "gqa_decode", "batch": 64, "cached": 4096, "ragged": True},
        # a 512-position block of a long prompt in the GQA layer (11,000 keys)
        {"name": "gqa_prompt_512_after_10488", "kind": "gqa_prompt", "tokens": 512, "before": 10488},
        # linear-attention layer: a prompt, then one decode step of 64 slots
        {"name": "gdn_prompt_4096", "kind": "gdn", "batch": 1, "tokens": 4096},
        {"name": "gdn_decode_64", "kind": "gdn", "batch": 64, "tokens": 1},
        # the reference-named calls an engine on host memory makes: next token, and a prompt in chunks of 512
        {"name": "engine_token_8191", "kind": "engine_token", "cached": 8191, "fp8": False},
        {"name": "engine_prompt_1100", "kind": "engine_prompt", "tokens": 1100},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["mla_decode", "mla_decode", "dsa_decode", "mla_prompt", "gqa_decode", "gqa_prompt", "gdn", "engine_token",
                       "engine_prompt"])
    if kind == "mla_decode":
        return {"kind": kind, "batch": _log(rng, 1, 64), "cached": _log(rng, 512, 32768), "ragged": rng.random() < 0.7}
    if kind == "dsa_decode":
        return {"kind": kind, "batch": _log(rng, 1, 8), "cached": _log(rng, 4096, 65536), "ragged": rng.random() < 0.7}
    if kind == "mla_prompt":
        n = _log(rng, 128, 4096)
        return {"kind": kind, "tokens": n, "before": 0 if rng.random() < 0.5 else rng.randint(1, 4096 - n) if n < 4096 else 0}
    if kind == "gqa_decode":
        return {"kind": kind, "batch": _log(rng, 1, 64), "cached": _log(rng, 256, 8192), "ragged": rng.random() < 0.7}
    if kind == "gqa_prompt":
        return {"kind": kind, "tokens": _log(rng, 128, 1024), "before": 0 if rng.random() < 0.3 else rng.randint(1, 10488)}
    if kind == "gdn":
        if rng.random() < 0.5:
            return {"kind": kind, "batch": 1, "tokens": _log(rng, 128, 4096)}
        return {"kind": kind, "batch": _log(rng, 1, 64), "tokens": 1}
    if kind == "engine_token":
        return {"kind": kind, "cached": _log(rng, 255, 8191), "fp8": rng.random() < 0.5}
    return {"kind": kind, "tokens": _log(rng, 64, 1100)}


def _lengths(case):
    """Cached tokens of each sequence: all alike, or spread over the upper half of the range (part of the case, not of the seed)."""
    B, T = case["batch"], case["cached"]
    if not case["ragged"]:
        return [T] * B
    spread = np.random.default_rng(1000 * B + T).integers(T // 2, T + 1, B)
    spread[-1] = T
    return [int(t) for t in spread]


class _State:
    pass


def _randn(gen, *shape, std=1.0):
    """bf16 N(0, std), made in slices so that a large cache needs no f32 copy of itself."""
    out = torch.empty(*shape, dtype=torch.bfloat16, device=DEV)
    flat = out.view(-1)
    step = 1 << 26
    for i in range(0, flat.numel(), step):
        part = flat[i:i + step]
        part.copy_(torch.randn(part.numel(), device=DEV, generator=gen) * std)
    return out


def _prepare_mla_decode(s, case, gen):
    B, T = case["batch"], case["cached"]
    s.q = _randn(gen, B, HEADS, LATENT + ROPE)
    s.cache = _randn(gen, B, T, LATENT + ROPE)
    s.kv_len = torch.tensor(_lengths(case), dtype=torch.int32, device=DEV)
    s.max_len = T


def _run_mla_decode(s):
    return s.attn.mla_decode(s.q, s.cache, s.kv_len, max_kv_len=s.max_len, scale=MLA_SCALE)


def _prepare_dsa_decode(s, case, gen):
    _prepare_mla_decode(s, case, gen)
    B, T = case["batch"], case["cached"]
    s.keys, s.kscale = synth.fp8_token_keys(B, T, IDX_DIM, gen, DEV)
    s.iq = torch.randn(B, IDX_HEADS, IDX_DIM, device=DEV, generator=gen).to(torch.bfloat16).float()
    s.iw = torch.rand(B, IDX_HEADS, device=DEV, generator=gen) / math.sqrt(IDX_DIM * IDX_HEADS)


def _run_dsa_decode(s):
    sel, nsel = s.attn.dsa_select(s.keys, s.kscale, s.iq, s.iw, s.kv_len, IDX_TOPK, False, max_n=s.max_len)
    out = s.attn.mla_decode(s.q, s.cache, nsel, sel=sel, scale=MLA_SCALE, max_kv_len=IDX_TOPK + 1)
    return {"out": out, "sel": sel, "nsel": nsel}


def _prepare_mla_prompt(s, case, gen):
    n, before = case["tokens"], case["before"]
    s.before = before

    def fp8(rows, cols):
        return synth.fp8_block128_weights(rows, cols, 0.02, gen, DEV)
    s.qa, s.qb, s.kva, s.o = (fp8(Q_LORA, HIDDEN), fp8(HEADS * (NOPE + ROPE), Q_LORA), fp8(LATENT + ROPE, HIDDEN),
                              fp8(HIDDEN, HEADS * VDIM))
    s.qa_n, s.kva_n = (1 + _randn(gen, Q_LORA, std=0.1)), (1 + _randn(gen, LATENT, std=0.1))
    s.wuk, s.wuv = _randn(gen, HEADS, NOPE, LATENT, std=0.02), _randn(gen, HEADS, VDIM, LATENT, std=0.02)
    s.x = _randn(gen, n, HIDDEN)
    s.cache = _randn(gen, before + n, LATENT + ROPE)
    # an engine's weights do not change: the context may keep its widened copies
    s.attn.ctx.check(s.attn.lib.cwk_ctx_weight_cache(s.attn.ctx.h, 1 << 30))


def _run_mla_prompt(s):
    att = s.attn.mla_prefill(s.x, *s.qa, *s.qb, *s.kva, s.qa_n, s.kva_n, s.wuk, s.cache, s.before, HEADS)
    y = s.attn.fp8_linear(s.attn.mla_unabsorb(att, s.wuv), *s.o, out_bf16=True)
    return {"attention": att, "y": y, "rows": s.cache[s.before:]}


def _prepare_gqa_decode(s, case, gen):
    B, T = case["batch"], case["cached"]
    s.q = _randn(gen, B, GQ_HEADS, GQ_DIM)
    s.k, s.v = _randn(gen, B, T, GQ_KV, GQ_DIM), _randn(gen, B, T, GQ_KV, GQ_DIM)
    s.kv_len = torch.tensor(_lengths(case), dtype=torch.int32, device=DEV)
    s.max_len = T


def _run_gqa_decode(s):
    return s.attn.gqa_decode(s.q, s.k, s.v, s.kv_len, max_kv_len=s.max_len)


def _prepare_gqa_prompt(s, case, gen):
    n, s.before = case["tokens"], case["before"]
    s.q = _randn(gen, n, GQ_HEADS, GQ_DIM)
    s.k, s.v = _randn(gen, s.before + n, GQ_KV, GQ_DIM), _randn(gen, s.before + n, GQ_KV, GQ_DIM)


def _run_gqa_prompt(s):
    return s.attn.gqa_prefill(s.q, s.k, s.v, s.before)


def _prepare_gdn(s, case, gen):
    B, n, nh, d = case["batch"], case["tokens"], GDN_HEADS, GDN_DIM
    key_dim, val_dim = nh // GDN_GROUP * d, nh * d

    def f32(*shape):
        return torch.randn(*shape, device=DEV, generator=gen)
    s.up = 0.1 * f32(B, n, 2 * key_dim + val_dim)
    kq = s.up[:, :, :2 * key_dim].view(B, n, 2 * key_dim // d, d)      # q and k heads come normalised
    kq /= kq.norm(dim=-1, keepdim=True)
    s.decay, s.beta, s.gate = f32(B, n, nh), f32(B, n, nh), f32(B, n, val_dim)
    s.a_log, s.dt_bias, s.norm = 0.5 * f32(nh), 0.5 * f32(nh), 1 + 0.1 * f32(d)
    s.S = 0.05 * f32(B, nh, d, d)


def _run_gdn(s):
    out = s.attn.gdn_scan(s.up, s.decay, s.beta, s.gate, s.a_log, s.dt_bias, s.norm, s.S, GDN_GROUP, 1e-6)
    return {"out": out, "state": s.S}


def _engine_layer(s, gen, fp8):
    """One layer of an engine whose weights, cache and activations live in host memory, in the reference's structs."""
    os.environ["CWICK_LATENT_BF16"] = "1"              # a serving engine's latent cache is bf16
    s.lib = lib.load()
    s.lib.cwk_dropin_reset()                           # another model: no mirror of an earlier one's weights
    s.keep = []

    def bf16(rows, cols, std):
        w = _randn(gen, rows, cols, std=std).view(torch.int16).cpu().numpy()
        s.keep.append(w)
        return compat.tensor(w, rows, cols)

    def proj(rows, cols):
        if not fp8:
            return bf16(rows, cols, 0.02)
        w, sc = synth.fp8_block128_weights(rows, cols, 0.02, gen, DEV)
        w, sc = w.cpu().numpy(), sc.cpu().numpy()
        s.keep += [w, sc]
        return compat.tensor_fp8(w, sc, rows, cols)
    qa, qb, kva = proj(Q_LORA, HIDDEN), proj(HEADS * NOPE, Q_LORA), proj(LATENT, HIDDEN)
    kvb, o = bf16(HEADS * (NOPE + VDIM), LATENT, 0.02), proj(HIDDEN, HEADS * VDIM)
    ones = np.full(max(Q_LORA, LATENT), 0x3F80, np.uint16)
    s.keep.append(ones)
    s.tensors = qa, qb, kva, kvb, o, compat.tensor(ones, 1, Q_LORA), compat.tensor(ones, 1, LATENT)
    s.spec = compat.make_spec(HIDDEN, HEADS, NOPE, VDIM, Q_LORA, LATENT, 1e-6)
    s.err = compat.Err()


def _engine_check(s, status=0):
    if status != 0 or s.err.status != 0:
        raise RuntimeError("status %d: %s" % (status or s.err.status, s.err.message.decode(errors="replace")))


def _prepare_engine_token(s, case, gen):
    _engine_layer(s, gen, case["fp8"])
    s.first = s.pos = case["cached"]
    s.cache = np.zeros((s.first + ENGINE_ROOM, LATENT), np.int16)
    s.cache[:s.first] = _randn(gen, s.first, LATENT).view(torch.int16).cpu().numpy()
    s.x = torch.randn(HIDDEN, device=DEV, generator=gen).cpu().numpy()
    s.fn = s.lib["cwick_attention_mla_decode"]         # (a function object of its own: its argument types are set here)
    s.fn.restype = None
    s.fn.argtypes = [C.c_void_p] * 11 + [C.c_int64] * 3 + [C.c_void_p] * 5


def _run_engine_token(s):
    """The sequence's next token; at the end of its room the sequence goes back to its prefix."""
    if s.pos == len(s.cache):
        s.pos = s.first
    qa, qb, kva, kvb, o, qa_n, kva_n = s.tensors
    out = np.empty(HIDDEN, np.float32)
    ref = C.byref
    s.fn(C.addressof(s.spec), ref(qa), ref(qb), ref(kva), ref(kvb), None, ref(o), ref(qa_n), ref(kva_n), s.cache.ctypes.data, None,
         len(s.cache), s.pos, 0, None, None, s.x.ctypes.data, out.ctypes.data, ref(s.err))
    _engine_check(s)
    s.pos += 1
    return {"out": out, "row": s.cache[s.pos - 1]}


def _prepare_engine_prompt(s, case, gen):
    _engine_layer(s, gen, False)                       # (the chunk call takes BF16 projections only)
    s.n = case["tokens"]
    s.cache = np.zeros((s.n, LATENT), np.int16)
    s.x = torch.randn(s.n, HIDDEN, device=DEV, generator=gen).cpu().numpy()
    s.out = np.zeros((s.n, HIDDEN), np.float32)
    s.fn = s.lib["cwick_attention_mla_prefill_chunk"]
    s.fn.restype = C.c_int
    s.fn.argtypes = [C.c_void_p] * 10 + [C.c_int64] * 4 + [C.c_void_p] * 5


def _run_engine_prompt(s):
    qa, qb, kva, kvb, o, qa_n, kva_n = s.tensors
    ref = C.byref
    for at in range(0, s.n, ENGINE_CHUNK):
        n = min(ENGINE_CHUNK, s.n - at)
        _engine_check(s, s.fn(C.addressof(s.spec), ref(qa), ref(qb), ref(kva), ref(kvb), ref(o), ref(qa_n), ref(kva_n), s.cache.ctypes.data,
                              None, s.n, at, n, 0, None, None, s.x[at:].ctypes.data, s.out[at:].ctypes.data, ref(s.err)))
    return {"out": s.out, "rows": s.cache}


_PREPARE = {"mla_decode": _prepare_mla_decode, "dsa_decode": _prepare_dsa_decode, "mla_prompt": _prepare_mla_prompt,
            "gqa_decode": _prepare_gqa_decode, "gqa_prompt": _prepare_gqa_prompt, "gdn": _prepare_gdn,
            "engine_token": _prepare_engine_token, "engine_prompt": _prepare_engine_prompt}
_RUN = {"mla_decode": _run_mla_decode, "dsa_decode": _run_dsa_decode, "mla_prompt": _run_mla_prompt, "gqa_decode": _run_gqa_decode,
        "gqa_prompt": _run_gqa_prompt, "gdn": _run_gdn, "engine_token": _run_engine_token, "engine_prompt": _run_engine_prompt}


def prepare(case, seed):
    s = _State()
    s.run = _RUN[case["kind"]]
    if not case["kind"].startswith("engine"):
        s.attn = Attn(0)
    _PREPARE[case["kind"]](s, case, torch.Generator(device=DEV).manual_seed(seed))
    return s


def run(state):
    return state.run(state)


def work(case):
    """Bytes: inputs once + outputs once. FLOPs: the contractions as the layer defines them."""
    kind = case["kind"]
    qkv = LATENT + ROPE
    if kind in ("mla_decode", "dsa_decode"):
        lens = _lengths(case)
        io = case["batch"] * HEADS * (qkv + LATENT) * 2
        if kind == "mla_decode":
            return {"bytes": sum(lens) * qkv * 2 + io, "flops": 2.0 * sum(lens) * HEADS * (qkv + LATENT)}
        rows = sum(min(t, IDX_TOPK) for t in lens)
        return {"bytes": sum(lens) * (IDX_DIM + 4) + rows * (qkv * 2 + 4) + io,
                "flops": 2.0 * sum(lens) * IDX_HEADS * IDX_DIM + 2.0 * rows * HEADS * (qkv + LATENT)}
    if kind == "mla_prompt":
        n, before = case["tokens"], case["before"]
        w8 = HIDDEN * Q_LORA + Q_LORA * HEADS * (NOPE + ROPE) + HIDDEN * qkv + HIDDEN * HEADS * VDIM
        w16 = HEADS * (NOPE + VDIM) * LATENT
        pairs = n * before + n * (n + 1) / 2.0
        return {"bytes": w8 + 2 * w16 + n * HIDDEN * 4 + n * HEADS * LATENT * 2 + (before + n) * qkv * 2,
                "flops": 2.0 * n * (w8 + w16) + 2.0 * pairs * HEADS * (NOPE + ROPE + LATENT)}
    if kind == "gqa_decode":
        lens = _lengths(case)
        return {"bytes": sum(lens) * GQ_KV * GQ_DIM * 4 + case["batch"] * GQ_HEADS * GQ_DIM * 4,
                "flops": 4.0 * sum(lens) * GQ_HEADS * GQ_DIM}
    if kind == "gqa_prompt":
        n, before = case["tokens"], case["before"]
        return {"bytes": (n + before) * GQ_KV * GQ_DIM * 4 + n * GQ_HEADS * GQ_DIM * 4,
                "flops": 4.0 * (n * before + n * (n + 1) / 2.0) * GQ_HEADS * GQ_DIM}
    if kind == "gdn":
        B, n, nh, d = case["batch"], case["tokens"], GDN_HEADS, GDN_DIM
        return {"bytes": 4 * B * (n * (2 * nh // GDN_GROUP * d + 3 * nh * d + 2 * nh) + 2 * nh * d * d),
                "flops": 6.0 * B * n * nh * d * d}
    proj = HIDDEN * Q_LORA + Q_LORA * HEADS * NOPE + HIDDEN * LATENT + HIDDEN * HEADS * VDIM
    kvb = HEADS * (NOPE + VDIM) * LATENT
    n, before = (1, case["cached"]) if kind == "engine_token" else (case["tokens"], 0)
    pairs = n * before + n * (n + 1) / 2.0
    return {"bytes": proj * (1 if case.get("fp8") else 2) + kvb * 2 + (before + n) * LATENT * 2 + n * HIDDEN * 8,
            "flops": 2.0 * n * (proj + kvb) + 4.0 * pairs * HEADS * LATENT}


def tolerance(case):
    if case["kind"] == "gdn":
        return {"rel": 2e-5}                           # f32 throughout; a prompt's sums may run in another order
    if case["kind"].startswith("engine"):
        return {"rel": 1e-2, "differ": 1e-2}           # bf16 attention between f32 projections; cache rows as bf16 bit patterns
    return {"rel": 1e-2}                               # bf16 operands and results; selected rows are exact
