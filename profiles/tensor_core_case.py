"""Small cases of the tcgen05 kernels and the small-step decode kernel for `ncu` captures: `python profiles/tensor_core_case.py NAME`

    prompt         fa_kernel: two prompts of 4096 tokens, 16 query over 8 kv heads
    window_prompt  fa_kernel: 4 x 2048 tokens over token-major cache rows, window 1024, distance bias
    latent         latent_decode_kernel: 64 single tokens over 3072 cached rows of 512 + 64, 16 heads
    experts        moe_rows_kernel: 8192 tokens x 4 of 32 experts, width 2048, feed-forward 768
    experts_few    moe_stream_kernel: the same of 64 tokens
    small_step     paged_decode_small_kernel: 4 rows of 1024 tokens, 16 over 8 heads
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


call = dict(prompt=prompt, window_prompt=window_prompt, latent=latent, experts=experts, experts_few=lambda: experts(64), small_step=small_step)[sys.argv[1]]()
for _ in range(4):
    o = call()
torch.cuda.synchronize()
print("ok", float(o.float().abs().mean()))
