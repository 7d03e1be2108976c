"""Small cases of the tensor-core kernels and of small steps for `ncu` captures: `python profiles/tensor_core_case.py NAME`

    prompt         fa_kernel: two prompts of 4096 tokens, 16 query over 8 kv heads
    window_prompt  fa_kernel: 4 x 2048 tokens over token-major cache rows, window 1024, distance bias
    window_step    window_attn_mma_kernel, key-sharing: 64 single tokens over 3072 rows, window 2048, 16 over 8 heads
    latent         latent_decode_kernel: 64 single tokens over 3072 cached rows of 512 + 64, 16 heads
    experts        moe_rows_kernel: 8192 tokens x 4 of 32 experts, width 2048, feed-forward 768
    experts_few    moe_stream_kernel: the same of 64 tokens
    small_step     paged_decode_small_kernel: 4 rows of 1024 tokens, 16 over 8 heads
    prompt_store   fa_kernel with the copies of K and V: 28 prompts of 561 tokens, 16 over 8 heads
    rows           linear_rows_kernel: 4 rows, gate_up of Qwen3-0.6B with add + norm in front and SiluAndMul behind
    router         moe_router_kernel: 8192 rows of 2048 columns, 40 outputs
    delta          channel_delta kernels: 4 x 2048 tokens, 16 heads of 128 x 128 over 4 query/key heads
"""
import os
import sys

import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "nano-vllm_b200"))

from nanovllm import mixops, ops  # noqa: E402
from nanovllm.layers.rotary_embedding import build_banded_cos_sin  # noqa: E402
from nanovllm.layers.window_attention import distance_slopes  # noqa: E402

dev = "cuda"
rnd = lambda *s: torch.randn(*s, device=dev).bfloat16()
cu = lambda S, n: torch.arange(0, S + 1, dtype=torch.int32, device=dev) * n


def prompt():
    q, k, v = rnd(8192, 16, 128), rnd(8192, 8, 128), rnd(8192, 8, 128)
    return lambda: ops.paged_prefill(0, q, k, v, cu(2, 4096), cu(2, 4096), 4096, 4096, 128 ** -0.5)


def window_prompt():
    q, cache = rnd(8192, 16 * 128), rnd(8192, 8 * 256)
    bt, sp = torch.arange(32, dtype=torch.int32, device=dev).view(4, 8), mixops.StepSpans(4, 2048, cu(4, 2048), cu(4, 2048), None)
    return lambda: mixops.window_attention(q, cache, bt, 256, sp, 16, 8, 128, 128, 0.088, distance_slopes(16, dev), 1024)


def window_step():
    q, cache = rnd(64, 16 * 128), rnd(64 * 3072, 8 * 256)
    bt = torch.arange(64 * 12, dtype=torch.int32, device=dev).view(64, 12)
    sp = mixops.StepSpans(64, 1, None, None, torch.full((64,), 3000, dtype=torch.int32, device=dev))
    return lambda: mixops.window_attention(q, cache, bt, 256, sp, 16, 8, 128, 128, 0.088, distance_slopes(16, dev), 2048)


def latent():
    n, L, R = 64, 3072, 512
    cache, q_lat, q_raw = rnd(n * L, R + 64), rnd(16, n, R), rnd(n, 16, 192)
    bt = torch.arange(n * L // 256, dtype=torch.int32, device=dev).view(n, -1)
    sp, cs = mixops.StepSpans(n, 1, None, None, torch.full((n,), L, dtype=torch.int32, device=dev)), build_banded_cos_sin(64, 4096, 1e4, None, dev)
    return lambda: mixops.latent_attention(q_lat, q_raw, 128, cache, bt, 256, sp, None, cs, 0.07)


def experts(n=8192):
    E, top, W, ff = 32, 4, 2048, 768
    h, w_in, w_out = rnd(n, W), rnd(E, 2 * ff, W), rnd(E, W, ff)
    idx = torch.rand(n, E, device=dev).topk(top).indices.int()
    wgt = torch.rand(n, top, device=dev)
    return lambda: mixops.moe_experts(h, idx, wgt, w_in, w_out, 2, False)


def small_step():
    ops.bind_kv_cache(torch.randn(ops.kv_cache_shape(1, 16, 8, 256, 128), device=dev).bfloat16())
    q, bt = rnd(4, 16, 128), torch.arange(16, dtype=torch.int32, device=dev).view(4, 4)
    ctx = torch.full((4,), 1024, dtype=torch.int32, device=dev)
    return lambda: ops.paged_decode(0, q, bt, ctx, 128 ** -0.5)


def prompt_store():
    ops.bind_kv_cache(torch.zeros(ops.kv_cache_shape(1, 64, 8, 256, 128), device=dev).bfloat16())
    q, k, v, slots = rnd(28 * 561, 16, 128), rnd(28 * 561, 8, 128), rnd(28 * 561, 8, 128), torch.arange(28 * 561, dtype=torch.int32, device=dev)
    return lambda: ops.paged_prefill_store(0, q, k, v, slots, cu(28, 561), cu(28, 561), 561, 561, 128 ** -0.5)


def rows():
    x, add, norm, w = rnd(4, 1024), rnd(4, 1024), rnd(1024), rnd(6144, 1024)
    return lambda: ops.linear_rows(x, w, norm, 1e-6, add, silu=True, pdl=True)[0]


def router():
    x, w = rnd(8192, 2048), torch.randn(40, 2048, device=dev)
    return lambda: mixops.moe_logits(x, w)


def delta():
    S, q, H, G, d = 4, 2048, 16, 4, 128
    x, write, z = rnd(S * q, (2 * G + H) * d), rnd(S * q, H), torch.randn(S * q, H * d, device=dev) - 4
    rate, bias, state = -torch.linspace(1, 16, H, device=dev), torch.zeros(H * d, device=dev), torch.zeros(S, H, d, d, device=dev)
    sp, slots = mixops.StepSpans(S, q, cu(S, q), cu(S, q), None), torch.arange(S, dtype=torch.int32, device=dev)
    return lambda: mixops.channel_state(x, 0, G * d, 2 * G * d, write, z, rate, bias, 1.0, state, slots, sp, H, G, d, d, d ** -0.5, forgetting=True)


call = dict(prompt=prompt, window_prompt=window_prompt, latent=latent, experts=experts, experts_few=lambda: experts(64), small_step=small_step,
            prompt_store=prompt_store, window_step=window_step, rows=rows, router=router, delta=delta)[sys.argv[1]]()
for _ in range(4):
    o = call()
torch.cuda.synchronize()
print("ok", float(o.float().abs().mean()))
