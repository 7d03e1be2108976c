"""Workloads of the framework with their sizes: what a program has it do, through its public entry points.

A case names a ``kind``:

  step      one decode step of Qwen3-0.6B (the benchmark's model), captured once and replayed, as the engine does: tokens in, logits out
  decode    the ``Attention`` operator on one token per sequence: append to the paged cache, attend over it
  prefill   the ``Attention`` operator on prompts: packed new prompts, or portions of prompts whose earlier keys are in the cache
  latent    the latent-attention layer (``LatentAttention``), prompts or single tokens
  window    the windowed grouped-query layer (``BiasedWindowAttention``), prompts or single tokens
  experts   a routed feed-forward (``RoutedExpertsFF`` / ``GroupRoutedExpertsFF``), a few tokens or a whole prompt step
  delta     the delta-rule layer with channel decays (``ChannelDeltaMixer``) on prompts

Sizes are those of the models under ``nanovllm/utils/synthetic.py`` and of the two widths the design benchmarks run; sequence lengths are spread
over ``lo`` to ``hi`` and put in an order by the seed, so batches are ragged.  Single-token layers are captured in a CUDA graph, as the engine captures its
decode step; prompt steps run eagerly, as the engine runs them.  Activations and weights are bf16; ``f32`` is the framework's fp32 format.
"""
from __future__ import annotations

import math
import os
import sys
from types import SimpleNamespace

import numpy as np
import torch
import torch.nn.functional as F

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nano-vllm_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from nanovllm import mixops, ops  # noqa: E402
from nanovllm.layers.attention import Attention  # noqa: E402
from nanovllm.layers.channel_state import ChannelDeltaMixer  # noqa: E402
from nanovllm.layers.latent_attention import LatentAttention  # noqa: E402
from nanovllm.layers.moe import GroupRoutedExpertsFF, RoutedExpertsFF  # noqa: E402
from nanovllm.layers.window_attention import BiasedWindowAttention  # noqa: E402
from nanovllm.models.qwen3 import Qwen3ForCausalLM  # noqa: E402
from nanovllm.utils.context import reset_context, set_context  # noqa: E402
from nanovllm.utils.synthetic import PRESETS, hf_config_dict  # noqa: E402

D = 128                  # head size of every attention here
EPS = 1e-6
PAGE = 256               # the engine's default page size
F64 = torch.float64


# ---- the cases -----------------------------------------------------------------------------------------------------------
def listed():
    return [
        # a few users: latency of a whole step is what they see, launches and small kernels are what it consists of
        dict(name="step_4_rows", kind="step", rows=4, lo=100, hi=1024, f32=False),
        # the benchmark's batch: 256 sequences, prompt and output between 100 and 1024 tokens, Qwen3-0.6B heads
        dict(name="decode_256_rows", kind="decode", rows=256, lo=100, hi=1024, heads=16, kv_heads=8, block=256, f32=False),
        # Qwen3-8B heads, pages of 16 (prefix cache), some long conversations in a small batch
        dict(name="decode_long_block16", kind="decode", rows=16, lo=600, hi=8192, heads=32, kv_heads=8, block=16, f32=False),
        # the benchmark's prompt step: as many prompts as fit 16384 tokens, packed
        dict(name="prefill_mix", kind="prefill", seqs=28, lo=100, hi=1024, prefix=0, heads=16, kv_heads=8, block=256, f32=False),
        # a portion of two long prompts (8192 tokens, scheduled in portions): the earlier half is in the cache
        dict(name="prefill_portion", kind="prefill", seqs=2, lo=4096, hi=4096, prefix=4096, heads=32, kv_heads=8, block=256, f32=False),
        # latent attention, a prompt step and a decode step
        dict(name="latent_prompts", kind="latent", decode=False, seqs=4, lo=2048, hi=2048, prefix=0, width=2048, f32=False),
        dict(name="latent_decode", kind="latent", decode=True, seqs=64, lo=2048, hi=4096, prefix=0, width=2048, f32=False),
        # windowed grouped-query attention, prompts of uneven lengths and a decode step
        dict(name="window_prompts", kind="window", decode=False, seqs=6, lo=500, hi=2200, prefix=0, width=2048, f32=False),
        dict(name="window_decode", kind="window", decode=True, seqs=64, lo=1024, hi=4096, prefix=0, width=2048, f32=False),
        # routed experts: a full prompt step, and a decode step of 64 rows
        dict(name="experts_prompts", kind="experts", tokens=8192, width=2048, grouped=True, f32=False),
        dict(name="experts_decode", kind="experts", tokens=64, width=2048, grouped=False, f32=False),
        # the delta rule over a prompt step: the serial one among the mixers
        dict(name="delta_prompts", kind="delta", seqs=4, lo=2048, hi=2048, width=2048, f32=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _span(rng, lo, hi, cap):
    """Two lengths lo <= hi, each over the logarithm of the range, hi at most cap."""
    hi_ = min(_log(rng, lo, hi), max(cap, lo))
    return max(lo, int(hi_ * rng.uniform(0.2, 1.0))), hi_


def draw(rng):
    kind = rng.choice(["step", "decode", "decode", "prefill", "prefill", "latent", "latent", "window", "window", "experts", "experts", "delta"])
    f32 = kind in ("latent", "window", "experts", "delta") and rng.random() < 0.12        # the fp32 format: small replays
    if kind == "step":
        lo, hi = _span(rng, 16, 1024, 1024)
        return dict(kind=kind, rows=_log(rng, 1, 64), lo=lo, hi=hi, f32=False)
    if kind == "decode":
        rows = _log(rng, 1, 256)
        lo, hi = _span(rng, 64, 8192, 260000 // rows)
        heads, kv = rng.choice([(16, 8), (32, 8), (8, 1)])
        return dict(kind=kind, rows=rows, lo=lo, hi=hi, heads=heads, kv_heads=kv, block=rng.choice([16, 256]), f32=False)
    if kind == "prefill":
        seqs = _log(rng, 1, 32)
        prefix = rng.choice([0, 0, _log(rng, 16, 4096)])
        lo, hi = _span(rng, 16, 8192, (8192 if prefix else 16384) // seqs)
        heads, kv = rng.choice([(16, 8), (32, 8), (8, 1)])
        return dict(kind=kind, seqs=seqs, lo=lo, hi=hi, prefix=prefix, heads=heads, kv_heads=kv, block=rng.choice([16, 256]), f32=False)
    width = rng.choice([1024, 2048])
    if kind in ("latent", "window"):
        if rng.random() < 0.5:
            seqs = _log(rng, 1, 8 if f32 else 128)
            lo, hi = _span(rng, 32, 8192, (4096 if f32 else 260000) // seqs)
            return dict(kind=kind, decode=True, seqs=seqs, lo=lo, hi=hi, prefix=0, width=width, f32=f32)
        seqs = _log(rng, 1, 4 if f32 else 16)
        lo, hi = _span(rng, 16, 4096, (512 if f32 else 8192) // seqs)
        prefix = 0 if f32 else rng.choice([0, 0, _log(rng, 16, 2048)])
        return dict(kind=kind, decode=False, seqs=seqs, lo=lo, hi=hi, prefix=prefix, width=width, f32=f32)
    if kind == "experts":
        return dict(kind=kind, tokens=_log(rng, 1, 256 if f32 else 8192), width=width, grouped=rng.random() < 0.5, f32=f32)
    seqs = _log(rng, 1, 4 if f32 else 16)
    lo, hi = _span(rng, 16, 4096, (1024 if f32 else 8192) // seqs)
    return dict(kind=kind, seqs=seqs, lo=lo, hi=hi, width=width, f32=f32)


# ---- shared pieces ---------------------------------------------------------------------------------------------------------
def _gen(seed, salt=0):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 1000003 + salt)


def _dtype(case):
    return torch.float32 if case["f32"] else torch.bfloat16


def _normal(g, *shape, std=1.0, dtype=torch.bfloat16):
    return (torch.randn(*shape, generator=g, device="cuda", dtype=torch.float32) * std).to(dtype)


def _grid(n, lo, hi):
    """n lengths spread evenly over [lo, hi]."""
    return [int(lo + (hi - lo) * (i + 0.5) / n) for i in range(n)]


def _lengths(n, lo, hi, seed):
    """The batch's lengths: the same ones for every seed, in the seed's order."""
    return [int(x) for x in np.random.default_rng(int(seed)).permutation(_grid(n, lo, hi))]


def _i32(a):
    return torch.tensor(np.asarray(a, dtype=np.int32), device="cuda")


def _tables(lens, block, seed, spare=0):
    """Page tables for sequences of these lengths over shuffled pages -> (int32 [n, width] with -1 behind the last page, pages in all)."""
    counts = [-(-n // block) for n in lens]
    total = sum(counts) + spare
    perm = np.random.default_rng(int(seed) + 17).permutation(total)
    bt = np.full((len(lens), max(counts)), -1, dtype=np.int32)
    at = 0
    for i, c in enumerate(counts):
        bt[i, :c] = perm[at:at + c]
        at += c
    return bt, total


def _slots(bt_row, block, a, b):
    p = np.arange(a, b)
    return bt_row[p // block].astype(np.int64) * block + p % block


def _captured(fn):
    """fn in a CUDA graph, as the engine keeps its decode step -> (graph, what fn returned)."""
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        fn()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = fn()
    return graph, out


def _replay(state):
    state.graph.replay()
    return state.out


def _spans(state):
    if state.decode:
        return mixops.StepSpans(len(state.lens), 1, None, None, _i32(state.lens))
    q, k = np.cumsum([0] + state.new), np.cumsum([0] + state.lens)
    return mixops.StepSpans(len(state.lens), max(state.new), _i32(q), _i32(k), None)


def _load(layer, weights):
    for leaf, w in weights.items():
        if not layer.load(leaf, w):
            raise KeyError(leaf)


def _rms(x, w):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS) * w.to(F64)


def _attend(q, k, v, scale, off, bias=None, window=0, sink=None):
    """float64 softmax attention of q [lq, H, d] over k [lk, G, d], v [lk, G, dv]; query i is at position off + i."""
    lq, H = q.shape[:2]
    lk, G = k.shape[:2]
    out = torch.empty(lq, H, v.shape[2], dtype=F64, device=q.device)
    j = torch.arange(lk, device=q.device)[None, :]
    for a in range(0, lq, 2048):
        i = off + torch.arange(a, min(a + 2048, lq), device=q.device)[:, None]
        hidden = (j > i) | ((i - j >= window) if window else (j > i))
        for h in range(H):
            s = q[a:a + 2048, h] @ k[:, h * G // H].T * scale
            if bias is not None:
                s -= bias[h] * (i - j)
            s.masked_fill_(hidden, -math.inf)
            if sink is not None:
                s = torch.cat((s, sink[h].expand(s.shape[0], 1)), -1)
            p = torch.softmax(s, -1)
            out[a:a + 2048, h] = p[:, :lk] @ v[:, h * G // H]
    return out


def _pairs(new, lens, window=0):
    """(query, key) pairs of causal attention, each query at the end of its keys."""
    total = 0.0
    for n, l in zip(new, lens):
        if window and l > window:
            first = max(l - n, 0)                       # position of the first query
            grow = max(0.0, min(window, l) - first)     # queries that see fewer than `window` keys
            total += grow * (first + 0.5 * (grow + 1)) + (n - grow) * window
        else:
            total += n * (l - n) + 0.5 * n * (n + 1)
    return total


# ---- paged grouped-query attention: the operator, and a whole decode step ----------------------------------------------------
_CACHE = {}


def _paged_cache(layers, blocks, kv_heads, block):
    """The process's bound KV cache, as an engine holds one: kept for the next states of its size, a layer (or a page range) for each."""
    key = (layers, blocks, kv_heads, block)
    if _CACHE.get("key") != key:
        _CACHE.clear()
        kv = torch.zeros(ops.kv_cache_shape(layers, blocks, kv_heads, block, D), dtype=torch.bfloat16, device="cuda")
        ops.bind_kv_cache(kv)
        _CACHE.update(key=key, kv=kv, turn=0)
    _CACHE["turn"] += 1
    return _CACHE["kv"], _CACHE["turn"] - 1


def _pool_blocks(case):
    """Pages for one state: the same for every seed, so that states share a cache."""
    n = case.get("rows") or case["seqs"]
    return n * -(-(case["hi"] + case.get("prefix", 0)) // case["block"])


def _paged_inputs(case, seed):
    g = _gen(seed)
    decode = case["kind"] == "decode"
    n, hq, hkv, block = case.get("rows") or case["seqs"], case["heads"], case["kv_heads"], case["block"]
    lens = _lengths(n, case["lo"], case["hi"], seed)
    new = [1] * n if decode else lens
    lens = [l + case.get("prefix", 0) for l in lens]
    bt, _ = _tables(lens, block, seed, spare=_pool_blocks(case) - sum(-(-l // block) for l in lens))
    s = SimpleNamespace(decode=decode, lens=lens, new=new, bt=bt, block=block, hq=hq, hkv=hkv)
    # queries and keys as the per-head norms leave them, side by side with the values in one projection
    s.qkv = _normal(g, sum(new), (hq + 2 * hkv) * D)
    old = (2, _pool_blocks(case), hkv, block, D)
    s.pages = torch.empty(old, dtype=torch.bfloat16, device="cuda").normal_(generator=g) if decode or case["prefix"] else None
    s.slot_mapping = np.concatenate([_slots(bt[i], block, l - m, l) for i, (l, m) in enumerate(zip(lens, new))])
    return s


def _paged_prepare(case, seed):
    s = _paged_inputs(case, seed)
    kv, turn = _paged_cache(8, _pool_blocks(case), s.hkv, s.block)
    layer = turn % 8
    pages = _pool_blocks(case)
    for i in range(2):
        kv[i, layer].zero_()
        if s.pages is not None:
            kv[i, layer, :pages].copy_(s.pages[i])
    s.pages = None
    s.attn = Attention(s.hq, D, D ** -0.5, s.hkv)
    s.attn.k_cache, s.attn.v_cache, s.attn.layer_id = kv[0, layer], kv[1, layer], layer
    n, a, b = s.qkv.shape[0], s.hq * D, (s.hq + s.hkv) * D
    s.q, s.k, s.v = s.qkv[:, :a].view(n, s.hq, D), s.qkv[:, a:b].view(n, s.hkv, D), s.qkv[:, b:].view(n, s.hkv, D)
    slots, bt = _i32(s.slot_mapping), _i32(s.bt)
    if s.decode:
        s.context = dict(is_prefill=False, slot_mapping=slots, context_lens=_i32(s.lens), block_tables=bt)
    else:
        s.context = dict(is_prefill=True, cu_seqlens_q=_i32(np.cumsum([0] + s.new)), cu_seqlens_k=_i32(np.cumsum([0] + s.lens)),
                         max_seqlen_q=max(s.new), max_seqlen_k=max(s.lens), slot_mapping=slots, block_tables=bt if case["prefix"] else None)
    return s


def _paged_run(s):
    set_context(**s.context)
    out = s.attn(s.q, s.k, s.v)
    reset_context()
    return {"out": out, "k_cache": s.attn.k_cache, "v_cache": s.attn.v_cache}


def _paged_exact(case, seed):
    s = _paged_inputs(case, seed)
    n, a, b = s.qkv.shape[0], s.hq * D, (s.hq + s.hkv) * D
    q, k, v = s.qkv[:, :a].view(n, s.hq, D).to(F64), s.qkv[:, a:b].view(n, s.hkv, D).to(F64), s.qkv[:, b:].view(n, s.hkv, D).to(F64)
    out, at = [], 0
    for i, (l, m) in enumerate(zip(s.lens, s.new)):
        kk, vv = k[at:at + m], v[at:at + m]
        if l > m:
            old = _slots(s.bt[i], s.block, 0, l - m)
            blk, row = torch.from_numpy(old // s.block).cuda(), torch.from_numpy(old % s.block).cuda()
            kk = torch.cat((s.pages[0][blk, :, row].to(F64), kk))
            vv = torch.cat((s.pages[1][blk, :, row].to(F64), vv))
        if s.decode:                                       # all heads of a key head at once: one query each
            G, r = s.hkv, s.hq // s.hkv
            p = torch.softmax(torch.einsum("grd,lgd->grl", q[at].view(G, r, D), kk) * D ** -0.5, -1)
            out.append(torch.einsum("grl,lgd->grd", p, vv).reshape(1, s.hq, D))
        else:
            out.append(_attend(q[at:at + m], kk, vv, D ** -0.5, l - m))
        at += m
    out = torch.cat(out)
    return {"out": out.unsqueeze(1) if s.decode else out, "k_cache": None, "v_cache": None}


def _paged_work(case):
    n, hq, hkv = case.get("rows") or case["seqs"], case["heads"], case["kv_heads"]
    lens = _grid(n, case["lo"], case["hi"])
    new = [1] * n if case["kind"] == "decode" else lens
    lens = [l + case.get("prefix", 0) for l in lens]
    t = sum(new)
    keys = sum(lens)
    rows = t * (2 * hq + 2 * hkv) + 2 * hkv * (keys if case["kind"] == "decode" or case["prefix"] else t)
    return {"bytes": 2 * D * rows, "flops": 4 * D * hq * _pairs(new, lens)}


QWEN = PRESETS["qwen3-0.6b"]
_MODEL = {}
STEP_SLOTS = 4           # page ranges of the step's cache: a state has one, the oldest gives way


def _qwen_weights():
    g = _gen(0, 1)
    H, inter, hq, hkv, V = (QWEN[k] for k in ("hidden_size", "intermediate_size", "num_attention_heads", "num_key_value_heads", "vocab_size"))
    yield "model.embed_tokens.weight", _normal(g, V, H, std=0.02)
    yield "model.norm.weight", 1 + _normal(g, H, std=0.1)
    for i in range(QWEN["num_hidden_layers"]):
        p = f"model.layers.{i}."
        for leaf, shape in (("self_attn.q_proj", (hq * D, H)), ("self_attn.k_proj", (hkv * D, H)), ("self_attn.v_proj", (hkv * D, H)),
                            ("self_attn.o_proj", (H, hq * D)), ("mlp.gate_proj", (inter, H)), ("mlp.up_proj", (inter, H)), ("mlp.down_proj", (H, inter))):
            yield p + leaf + ".weight", _normal(g, *shape, std=0.02)
        for leaf, cols in (("input_layernorm", H), ("post_attention_layernorm", H), ("self_attn.q_norm", D), ("self_attn.k_norm", D)):
            yield p + leaf + ".weight", 1 + _normal(g, cols, std=0.1)


def _qwen_model():
    """The model a serving process holds: loaded once."""
    if not _MODEL:
        model = Qwen3ForCausalLM(SimpleNamespace(**hf_config_dict(QWEN)), 0, 1, "cuda", max_position=4096)
        for name, w in _qwen_weights():
            model.load_hf_tensor(name, w)
        _MODEL["model"] = model
    return _MODEL["model"]


def _step_inputs(case, seed):
    g = _gen(seed)
    rows = case["rows"]
    lens = _lengths(rows, case["lo"], case["hi"], seed)
    pool = rows * -(-case["hi"] // PAGE)
    bt, _ = _tables(lens, PAGE, seed, spare=pool - sum(-(-l // PAGE) for l in lens))
    ids = torch.randint(0, QWEN["vocab_size"], (rows,), generator=g, device="cuda")
    shape = (2, QWEN["num_hidden_layers"], pool, QWEN["num_key_value_heads"], PAGE, D)
    pages = torch.empty(shape, dtype=torch.bfloat16, device="cuda").normal_(generator=g)
    return SimpleNamespace(lens=lens, bt=bt, ids=ids, pages=pages, pool=pool)


def _step_prepare(case, seed):
    s = _step_inputs(case, seed)
    model = _qwen_model()
    kv, turn = _paged_cache(QWEN["num_hidden_layers"], STEP_SLOTS * s.pool, model.num_kv_heads, PAGE)
    base = (turn % STEP_SLOTS) * s.pool
    kv[:, :, base:base + s.pool].copy_(s.pages)
    s.pages = None
    for i, a in enumerate(model.modules()):
        a.k_cache, a.v_cache, a.layer_id = kv[0, i], kv[1, i], i
    bt = np.where(s.bt >= 0, s.bt + base, -1)
    positions = torch.tensor([l - 1 for l in s.lens], dtype=torch.int64, device="cuda")
    context = dict(is_prefill=False, context_lens=_i32(s.lens), block_tables=_i32(bt),
                   slot_mapping=_i32([_slots(bt[i], PAGE, l - 1, l)[0] for i, l in enumerate(s.lens)]))

    def step():
        set_context(**context)
        logits = model.compute_logits(model(s.ids, positions))
        reset_context()
        return logits

    s.keep = (context, positions)
    s.graph, s.out = _captured(step)
    return s


def _step_exact(case, seed):
    s = _step_inputs(case, seed)
    W = dict(_qwen_weights())
    n, hq, hkv = len(s.lens), QWEN["num_attention_heads"], QWEN["num_key_value_heads"]
    pos = torch.tensor([l - 1 for l in s.lens], dtype=F64, device="cuda")
    ang = pos[:, None] * (1e6 ** (-torch.arange(0, D, 2, dtype=F64, device="cuda") / D))[None]
    cos, sin = ang.cos()[:, None], ang.sin()[:, None]

    def rotate(x):
        a, b = x[..., :D // 2], x[..., D // 2:]
        return torch.cat((a * cos - b * sin, b * cos + a * sin), -1)

    x = W["model.embed_tokens.weight"][s.ids].to(F64)
    for i in range(QWEN["num_hidden_layers"]):
        w = lambda leaf: W[f"model.layers.{i}.{leaf}.weight"].to(F64)
        h = _rms(x, w("input_layernorm"))
        q = rotate(_rms((h @ w("self_attn.q_proj").T).view(n, hq, D), w("self_attn.q_norm")))
        k = rotate(_rms((h @ w("self_attn.k_proj").T).view(n, hkv, D), w("self_attn.k_norm")))
        v = (h @ w("self_attn.v_proj").T).view(n, hkv, D)
        o = []
        for r, l in enumerate(s.lens):
            old = _slots(s.bt[r], PAGE, 0, l - 1)
            blk, row = torch.from_numpy(old // PAGE).cuda(), torch.from_numpy(old % PAGE).cuda()
            kk = torch.cat((s.pages[0, i][blk, :, row].to(F64), k[r:r + 1]))
            vv = torch.cat((s.pages[1, i][blk, :, row].to(F64), v[r:r + 1]))
            p = torch.softmax(torch.einsum("grd,lgd->grl", q[r].view(hkv, hq // hkv, D), kk) * D ** -0.5, -1)
            o.append(torch.einsum("grl,lgd->grd", p, vv).reshape(hq * D))
        x = x + torch.stack(o) @ w("self_attn.o_proj").T
        h = _rms(x, w("post_attention_layernorm"))
        x = x + (F.silu(h @ w("mlp.gate_proj").T) * (h @ w("mlp.up_proj").T)) @ w("mlp.down_proj").T
    return _rms(x, W["model.norm.weight"]) @ W["model.embed_tokens.weight"].to(F64).T


def _step_work(case):
    rows, H, L = case["rows"], QWEN["hidden_size"], QWEN["num_hidden_layers"]
    hq, hkv, inter, V = QWEN["num_attention_heads"], QWEN["num_key_value_heads"], QWEN["intermediate_size"], QWEN["vocab_size"]
    layer = H * D * (hq + 2 * hkv) + H * D * hq + 3 * H * inter
    keys = sum(_grid(rows, case["lo"], case["hi"]))
    return {"bytes": 2 * (L * layer + V * H + rows * V) + L * keys * 4 * hkv * D,
            "flops": 2 * rows * (L * layer + V * H) + 4 * L * keys * hq * D}


# ---- latent attention ----------------------------------------------------------------------------------------------------------
def _latent_dims(width):
    rank = width // 4
    return dict(heads=16, dim=128, rot_dim=64, vdim=128, kv_rank=rank, q_rank=3 * rank // 2, scale=192 ** -0.5, rot={"base": 1e6, "dims": 64})


def _latent_inputs(case, seed):
    g, dt, width = _gen(seed), _dtype(case), case["width"]
    m = _latent_dims(width)
    H, d, rd, vd, R, Q = (m[k] for k in ("heads", "dim", "rot_dim", "vdim", "kv_rank", "q_rank"))
    lens = _lengths(case["seqs"], case["lo"], case["hi"], seed)
    new = [1] * len(lens) if case["decode"] else lens
    lens = [l + case["prefix"] for l in lens]
    s = SimpleNamespace(decode=case["decode"], lens=lens, new=new, m=m)
    s.weights = {"dq": _normal(g, Q, width, std=width ** -0.5, dtype=dt), "dkv": _normal(g, R + rd, width, std=width ** -0.5, dtype=dt),
                 "dq.norm": 1 + _normal(g, Q, std=0.1, dtype=dt), "dkv.norm": 1 + _normal(g, R, std=0.1, dtype=dt),
                 "uq": _normal(g, H * (d + rd), Q, std=Q ** -0.5, dtype=dt), "uk": _normal(g, H * d, R, std=R ** -0.5, dtype=dt),
                 "uv": _normal(g, H * vd, R, std=R ** -0.5, dtype=dt), "o": _normal(g, width, H * vd, std=(H * vd) ** -0.5, dtype=dt),
                 "sink": _normal(g, H, dtype=torch.float32)}
    s.h = _normal(g, sum(new), width, dtype=dt)
    s.old = [_normal(g, l - n, R + rd, dtype=dt) for l, n in zip(lens, new)]      # rows of earlier tokens: normed latent, rotated key part
    s.bt, s.blocks = _tables(lens, PAGE, seed)
    return s


def _fill_rows(cache, s):
    for i, rows in enumerate(s.old):
        if rows.shape[0]:
            cache[torch.from_numpy(_slots(s.bt[i], PAGE, 0, rows.shape[0])).cuda()] = rows


def _layer_context(s, state_slots=None):
    return SimpleNamespace(block_tables=_i32(s.bt), state_slots=state_slots,
                           slot_mapping=_i32(np.concatenate([_slots(s.bt[i], PAGE, l - n, l) for i, (l, n) in enumerate(zip(s.lens, s.new))])))


def _positions(s):
    return torch.from_numpy(np.concatenate([np.arange(l - n, l) for l, n in zip(s.lens, s.new)]).astype(np.int64)).cuda()


def _latent_prepare(case, seed):
    s = _latent_inputs(case, seed)
    s.layer = LatentAttention(case["width"], s.m, EPS, _dtype(case), "cuda", 16384)
    _load(s.layer, s.weights)
    s.layer.block_size = PAGE
    s.layer.cache = torch.zeros(s.blocks * PAGE, s.layer.cache_row_elems(), dtype=_dtype(case), device="cuda")
    _fill_rows(s.layer.cache, s)
    s.weights = s.old = None
    s.ctx, s.spans, s.positions = _layer_context(s), _spans(s), _positions(s)
    s.call = lambda: {"out": s.layer.forward(s.h, s.positions, s.ctx, s.spans), "cache": s.layer.cache}
    if s.decode:
        s.graph, s.out = _captured(s.call)
    return s


def _layer_run(s):
    return _replay(s) if s.decode else s.call()


def _latent_exact(case, seed):
    s = _latent_inputs(case, seed)
    m, W = s.m, {k: w.to(F64) for k, w in s.weights.items()}
    H, d, rd, vd, R = (m[k] for k in ("heads", "dim", "rot_dim", "vdim", "kv_rank"))
    h = s.h.to(F64)
    ang = _positions(s).to(F64)[:, None] * (1e6 ** (-torch.arange(0, rd, 2, dtype=F64, device="cuda") / rd))[None]

    def rotate(x, cos, sin):
        a, b = x[..., 0::2], x[..., 1::2]
        return torch.stack((a * cos - b * sin, b * cos + a * sin), -1).flatten(-2)

    q = (_rms(h @ W["dq"].T, W["dq.norm"]) @ W["uq"].T).view(-1, H, d + rd)
    q = torch.cat((q[..., :d], rotate(q[..., d:], ang.cos()[:, None], ang.sin()[:, None])), -1)
    kv = h @ W["dkv"].T
    rows = torch.cat((_rms(kv[:, :R], W["dkv.norm"]), rotate(kv[:, R:], ang.cos(), ang.sin())), -1)
    out, at = torch.empty(h.shape[0], H, vd, dtype=F64, device="cuda"), 0
    uk, uv = W["uk"].view(H, d, R), W["uv"].view(H, vd, R)
    for i, (l, n) in enumerate(zip(s.lens, s.new)):
        c = torch.cat((s.old[i].to(F64), rows[at:at + n]))
        for a in range(0, H, 4):                           # a few heads at a time: their keys and values are wide
            k = torch.cat((torch.einsum("lr,hdr->lhd", c[:, :R], uk[a:a + 4]), c[:, None, R:].expand(-1, 4, -1)), -1)
            v = torch.einsum("lr,hdr->lhd", c[:, :R], uv[a:a + 4])
            out[at:at + n, a:a + 4] = _attend(q[at:at + n, a:a + 4], k, v, m["scale"], l - n, sink=W["sink"][a:a + 4])
        at += n
    return {"out": out.flatten(1) @ W["o"].T, "cache": None}


def _latent_work(case):
    m, width, e = _latent_dims(case["width"]), case["width"], 4 if case["f32"] else 2
    H, d, rd, vd, R, Q = (m[k] for k in ("heads", "dim", "rot_dim", "vdim", "kv_rank", "q_rank"))
    lens = _grid(case["seqs"], case["lo"], case["hi"])
    new = [1] * len(lens) if case["decode"] else lens
    lens = [l + case["prefix"] for l in lens]
    t, keys, pairs = sum(new), sum(lens), _pairs(new, lens)
    weights = (Q + R + rd) * width + H * (d + rd) * Q + H * (d + vd) * R + width * H * vd
    # per head the scores and values either meet the latents themselves, or keys and values formed from them
    latents = H * (pairs * (2 * R + rd) + t * R * (d + vd))
    formed = H * (pairs * (d + rd + vd) + keys * R * (d + vd))
    return {"bytes": e * (weights + 2 * t * width + (keys + t) * (R + rd)),
            "flops": 2 * (t * ((Q + R + rd) * width + H * (d + rd) * Q + width * H * vd) + min(latents, formed))}


# ---- windowed grouped-query attention ---------------------------------------------------------------------------------------------
def _window_dims(width):
    return dict(heads=16, kv_heads=8, dim=D, vdim=D, scale=D ** -0.5, mask={"size": width})


def _window_inputs(case, seed):
    g, dt, width = _gen(seed), _dtype(case), case["width"]
    m = _window_dims(width)
    H, G = m["heads"], m["kv_heads"]
    lens = _lengths(case["seqs"], case["lo"], case["hi"], seed)
    new = [1] * len(lens) if case["decode"] else lens
    lens = [l + case["prefix"] for l in lens]
    s = SimpleNamespace(decode=case["decode"], lens=lens, new=new, m=m)
    s.weights = {"q": _normal(g, H * D, width, std=width ** -0.5, dtype=dt), "k": _normal(g, G * D, width, std=width ** -0.5, dtype=dt),
                 "v": _normal(g, G * D, width, std=width ** -0.5, dtype=dt), "q.norm": 1 + _normal(g, H * D, std=0.1, dtype=dt),
                 "k.norm": 1 + _normal(g, G * D, std=0.1, dtype=dt), "o": _normal(g, width, H * D, std=(H * D) ** -0.5, dtype=dt)}
    s.h = _normal(g, sum(new), width, dtype=dt)
    s.old = [_normal(g, l - n, 2 * G * D, dtype=dt) for l, n in zip(lens, new)]
    s.bt, s.blocks = _tables(lens, PAGE, seed)
    return s


def _window_prepare(case, seed):
    s = _window_inputs(case, seed)
    s.layer = BiasedWindowAttention(case["width"], s.m, EPS, _dtype(case), "cuda")
    _load(s.layer, s.weights)
    s.layer.block_size = PAGE
    s.layer.cache = torch.zeros(s.blocks * PAGE, s.layer.cache_row_elems(), dtype=_dtype(case), device="cuda")
    _fill_rows(s.layer.cache, s)
    s.weights = s.old = None
    s.ctx, s.spans = _layer_context(s), _spans(s)
    s.call = lambda: {"out": s.layer.forward(s.h, s.ctx, s.spans), "cache": s.layer.cache}
    if s.decode:
        s.graph, s.out = _captured(s.call)
    return s


def _window_exact(case, seed):
    s = _window_inputs(case, seed)
    m, W, h = s.m, {k: w.to(F64) for k, w in s.weights.items()}, s.h.to(F64)
    H, G = m["heads"], m["kv_heads"]
    q = _rms(h @ W["q"].T, W["q.norm"]).view(-1, H, D)
    k, v = _rms(h @ W["k"].T, W["k.norm"]), h @ W["v"].T
    slopes = torch.exp2(-8.0 * torch.arange(1, H + 1, dtype=F64) / H).cuda()
    out, at = [], 0
    for i, (l, n) in enumerate(zip(s.lens, s.new)):
        old = s.old[i].to(F64)
        kk, vv = torch.cat((old[:, :G * D], k[at:at + n])).view(l, G, D), torch.cat((old[:, G * D:], v[at:at + n])).view(l, G, D)
        out.append(_attend(q[at:at + n], kk, vv, m["scale"], l - n, bias=slopes, window=m["mask"]["size"]))
        at += n
    return {"out": torch.cat(out).flatten(1) @ W["o"].T, "cache": None}


def _window_work(case):
    m, width, e = _window_dims(case["width"]), case["width"], 4 if case["f32"] else 2
    H, G, window = m["heads"], m["kv_heads"], m["mask"]["size"]
    lens = _grid(case["seqs"], case["lo"], case["hi"])
    new = [1] * len(lens) if case["decode"] else lens
    lens = [l + case["prefix"] for l in lens]
    t = sum(new)
    seen = sum(min(l, window + n - 1) for l, n in zip(lens, new))
    weights = width * D * (2 * H + 2 * G)
    return {"bytes": e * (weights + 2 * t * width + (seen + t) * 2 * G * D),
            "flops": 2 * t * weights + 4 * D * H * _pairs(new, lens, window)}


# ---- routed experts ---------------------------------------------------------------------------------------------------------------
def _experts_dims(case):
    width = case["width"]
    E, top = (16, 2) if width == 1024 else (32, 4)
    m = {"router": {"experts": E, "top": top}, "expert": {"ff": 3 * width // (2 * top)}, "shared": {"ff": width}}
    if case["grouped"]:
        m["router"].update({"identity": E // 4, "scale": 2.0, "groups": {"count": 4 if width == 1024 else 8, "keep": 2 if width == 1024 else 4}})
    return m


def _experts_inputs(case, seed):
    g, dt, width = _gen(seed), _dtype(case), case["width"]
    m = _experts_dims(case)
    E, ff, sff = m["router"]["experts"], m["expert"]["ff"], m["shared"]["ff"]
    outs = E + m["router"].get("identity", 0)
    s = SimpleNamespace(m=m)
    s.x32 = torch.randn(case["tokens"], width, generator=g, device="cuda")
    s.h = s.x32.to(dt)
    s.weights = {"router": _normal(g, outs, width, std=width ** -0.5, dtype=torch.float32)}
    names = ("gate", "up") if case["grouped"] else ("up",)
    for k in range(E):
        for name in names:
            s.weights[f"e{k}.{name}"] = _normal(g, ff, width, std=width ** -0.5, dtype=dt)
        s.weights[f"e{k}.down"] = _normal(g, width, ff, std=ff ** -0.5, dtype=dt)
    for name in names:
        s.weights["shared." + name] = _normal(g, sff, width, std=width ** -0.5, dtype=dt)
    s.weights["shared.down"] = _normal(g, width, sff, std=sff ** -0.5, dtype=dt)
    if case["grouped"]:
        s.weights["correction"] = _normal(g, outs, std=0.01, dtype=torch.float32)
    else:
        s.weights["shared.sg"] = _normal(g, 1, width, std=width ** -0.5, dtype=torch.float32)
    return s


def _experts_prepare(case, seed):
    s = _experts_inputs(case, seed)
    s.layer = (GroupRoutedExpertsFF if case["grouped"] else RoutedExpertsFF)(case["width"], s.m, _dtype(case), "cuda")
    _load(s.layer, s.weights)
    s.weights = None
    s.call = (lambda: s.layer.forward(s.h, s.x32)) if case["grouped"] else (lambda: s.layer.forward(s.h)[1])
    s.decode = case["tokens"] <= 256                        # a decode step: captured; a prompt step runs eagerly
    if s.decode:
        s.graph, s.out = _captured(s.call)
    return s


def _experts_exact(case, seed):
    s = _experts_inputs(case, seed)
    m, W, r = s.m, s.weights, s.m["router"]
    E, top = r["experts"], r["top"]
    w = lambda leaf: W[leaf].to(F64)
    h = s.h.to(F64)
    if case["grouped"]:
        x = s.x32.to(F64)
        p = torch.softmax(x @ w("router").T, -1)
        c = p + w("correction")
        n, outs, count, keep = p.shape[0], p.shape[1], r["groups"]["count"], r["groups"]["keep"]
        per = c.view(n, count, outs // count)
        best = per.max(-1).values.topk(keep, -1).indices
        shut = torch.ones(n, count, dtype=torch.bool, device="cuda").scatter_(1, best, False)
        chosen = per.masked_fill(shut[:, :, None], -math.inf).reshape(n, outs).topk(top, -1).indices
        weight = p.gather(1, chosen)
        weight = weight / (weight.sum(-1, keepdim=True) + 1e-20) * r["scale"]
        out = (F.silu(h @ w("shared.gate").T) * (h @ w("shared.up").T)) @ w("shared.down").T
        out += (weight * (chosen >= E)).sum(-1, keepdim=True) * x
    else:
        p = torch.sigmoid(h @ w("router").T)
        weight, chosen = p.topk(top, -1)
        out = torch.relu(h @ w("shared.up").T).square() @ w("shared.down").T * torch.sigmoid(h @ w("shared.sg").T)
    for k in range(E):
        t, at = (chosen == k).nonzero(as_tuple=True)
        if case["grouped"]:
            y = (F.silu(h[t] @ w(f"e{k}.gate").T) * (h[t] @ w(f"e{k}.up").T)) @ w(f"e{k}.down").T * weight[t, at, None]
        else:
            y = torch.relu(h[t] * weight[t, at, None] @ w(f"e{k}.up").T).square() @ w(f"e{k}.down").T
        out.index_add_(0, t, y)
    return out


def _experts_work(case):
    m, width, n, e = _experts_dims(case), case["width"], case["tokens"], 4 if case["f32"] else 2
    r, parts = m["router"], 3 if case["grouped"] else 2
    outs = r["experts"] + r.get("identity", 0)
    real = n * r["top"] * r["experts"] / outs              # (token, expert) pairs whose expert has tensors
    touched = r["experts"] * (1 - (1 - r["top"] / outs) ** n)
    one, shared = parts * width * m["expert"]["ff"], parts * width * m["shared"]["ff"]
    return {"bytes": e * (touched * one + shared + n * width) + 4 * (outs * width + n * width * (2 if case["grouped"] else 1)),
            "flops": 2 * (real * one + n * (shared + outs * width))}


# ---- the delta rule with channel decays --------------------------------------------------------------------------------------------
def _delta_dims(width):
    return dict(heads=width // 128, kv_heads=4, dim=128, vdim=128, conv=4)


def _delta_inputs(case, seed):
    g, dt, width = _gen(seed), _dtype(case), case["width"]
    m = _delta_dims(width)
    H, G, d, vd = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
    lens = _lengths(case["seqs"], case["lo"], case["hi"], seed)
    s = SimpleNamespace(decode=False, lens=lens, new=lens, m=m)
    lin = lambda rows, cols: _normal(g, rows, cols, std=cols ** -0.5, dtype=dt)
    step = torch.exp(torch.empty(H * d, device="cuda").uniform_(math.log(1e-3), math.log(0.1), generator=g))
    s.weights = {"q": lin(G * d, width), "k": lin(G * d, width), "v": lin(H * vd, width), "b": lin(H, width), "a1": lin(d, width), "g1": lin(d, width),
                 "a2": lin(H * d, d), "g2": lin(H * vd, d), "q.conv": _normal(g, G * d, 4, std=0.5, dtype=dt),
                 "k.conv": _normal(g, G * d, 4, std=0.5, dtype=dt), "v.conv": _normal(g, H * vd, 4, std=0.5, dtype=dt),
                 "A_log": torch.log(torch.empty(H, device="cuda").uniform_(1.0, 16.0, generator=g)),
                 "dt_bias": step + torch.log(-torch.expm1(-step)), "norm": 1 + _normal(g, vd, std=0.1, dtype=dt), "o": lin(width, H * vd)}
    s.h = _normal(g, sum(lens), width, dtype=dt)
    return s


def _delta_prepare(case, seed):
    s = _delta_inputs(case, seed)
    m, n = s.m, len(s.lens)
    s.layer = ChannelDeltaMixer(case["width"], m, EPS, _dtype(case), "cuda", ranks={"a1": m["dim"], "g1": m["dim"]})
    _load(s.layer, s.weights)
    s.weights = None
    s.layer.bind(0, PAGE, n)
    s.ctx = SimpleNamespace(state_slots=_i32(np.random.default_rng(seed).permutation(n)))
    s.spans = _spans(s)
    s.call = lambda: {"out": s.layer.forward(s.h, None, s.ctx, s.spans), "state": s.layer.state[0], "conv": s.layer.conv_state[0]}
    return s


def _delta_exact(case, seed):
    s = _delta_inputs(case, seed)
    m, W = s.m, {k: w.to(F64) for k, w in s.weights.items()}
    H, G, d, vd, n = m["heads"], m["kv_heads"], m["dim"], m["vdim"], len(s.lens)
    order = sorted(range(n), key=lambda i: -s.lens[i])     # the longest first: the sequences still running are the first ones
    top = max(s.lens)
    h = torch.zeros(n, top, case["width"], dtype=F64, device="cuda")
    at = np.cumsum([0] + s.lens)
    for r, i in enumerate(order):
        h[r, :s.lens[i]] = s.h[at[i]:at[i + 1]].to(F64)

    def conv(leaf):
        x, w = h @ W[leaf].T, W[leaf + ".conv"]
        y = x * w[:, 3]
        for j in range(1, 4):
            y[:, j:] += x[:, :-j] * w[:, 3 - j]
        return F.silu(y)

    unit = lambda x: x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)
    per = lambda x: x.view(n, top, G, d).repeat_interleave(H // G, 2)
    q, k = per(unit(conv("q").view(n, top, G, d)) * d ** -0.5), per(unit(conv("k").view(n, top, G, d)))
    v, beta = conv("v").view(n, top, H, vd), torch.sigmoid(h @ W["b"].T)
    z = (h @ W["a1"].T @ W["a2"].T + W["dt_bias"]).view(n, top, H, d)
    decay = torch.exp(-torch.exp(W["A_log"])[:, None] * F.softplus(z))
    S, o = torch.zeros(n, H, vd, d, dtype=F64, device="cuda"), torch.zeros(n, top, H, vd, dtype=F64, device="cuda")
    running = [sum(l > t for l in s.lens) for t in range(top)]
    for t in range(top):
        r = running[t]
        St = S[:r]
        St *= decay[:r, t, :, None]
        u = beta[:r, t, :, None] * (v[:r, t] - torch.matmul(St, k[:r, t, :, :, None])[..., 0])
        St += u[..., None] * k[:r, t, :, None]
        o[:r, t] = torch.matmul(St, q[:r, t, :, :, None])[..., 0]
    y = _rms(o, W["norm"]).flatten(2) * torch.sigmoid(h @ W["g1"].T @ W["g2"].T)
    y = y @ W["o"].T
    out = torch.empty(at[-1], case["width"], dtype=F64, device="cuda")
    slots = np.random.default_rng(seed).permutation(n)
    state = torch.empty_like(S)
    for r, i in enumerate(order):
        out[at[i]:at[i + 1]] = y[r, :s.lens[i]]
        state[slots[i]] = S[r]
    return {"out": out, "state": state, "conv": None}


def _delta_work(case):
    m, width, e = _delta_dims(case["width"]), case["width"], 4 if case["f32"] else 2
    H, G, d, vd = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
    t = sum(_grid(case["seqs"], case["lo"], case["hi"]))
    weights = width * (2 * G * d + H * vd + H + 2 * d) + d * H * (d + vd) + width * H * vd
    # decay, read-out against the key, the write and the read-out against the query: 7 operations per state element and token
    return {"bytes": e * (weights + 2 * t * width) + 4 * case["seqs"] * H * d * vd, "flops": 2 * t * weights + 7 * t * H * d * vd}


# ---- the file's interface ------------------------------------------------------------------------------------------------------------
_KINDS = {
    "step": (_step_prepare, _replay, _step_exact, _step_work),
    "decode": (_paged_prepare, _paged_run, _paged_exact, _paged_work),
    "prefill": (_paged_prepare, _paged_run, _paged_exact, _paged_work),
    "latent": (_latent_prepare, _layer_run, _latent_exact, _latent_work),
    "window": (_window_prepare, _layer_run, _window_exact, _window_work),
    "experts": (_experts_prepare, _layer_run, _experts_exact, _experts_work),
    "delta": (_delta_prepare, _layer_run, _delta_exact, _delta_work),
}


def prepare(case, seed):
    with torch.no_grad():
        state = _KINDS[case["kind"]][0](case, seed)
    state.kind = case["kind"]
    return state


def run(state):
    with torch.no_grad():
        return _KINDS[state.kind][1](state)


def exact(case, seed):
    with torch.no_grad():
        return _KINDS[case["kind"]][2](case, seed)


def work(case):
    return _KINDS[case["kind"]][3](case)


# Largest relative error another correct implementation would show, in bf16 and in fp32: about four times what the paths' error against
# ``exact`` measures on a B200.  Rounding travels through all 28 layers of the whole step.
_TOLERANCE = {"step": (0.1, None), "decode": (0.01, None), "prefill": (0.01, None), "latent": (0.02, 1e-5), "window": (0.015, 1e-5),
              "experts": (0.012, 1e-5), "delta": (0.015, 1e-5)}


def tolerance(case):
    return {"rel": _TOLERANCE[case["kind"]][1 if case["f32"] else 0]}
