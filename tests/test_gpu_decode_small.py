"""Paged decode of small steps (csrc/decode_small.cu): one CTA and clusters of 2, 4 and 8 per context, every head group, contexts around chunk
and page edges, empty rows, stale rows, and the fused form's append.  Tolerance as the other decode tests."""
import pytest
import torch

from oracle.paged_attention_ref import paged_decode_ref, to_logical
from oracle.qwen3_ref import rmsnorm_ref, rope_ref, rope_table
from test_gpu_kernels import assert_close_bf16, bf, bind_random_cache, make_tables

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from nanovllm import ops as _ops
    return _ops


@pytest.mark.parametrize("hq,hkv", [(2, 2), (4, 2), (8, 2), (16, 2)])
@pytest.mark.parametrize("bs,lens", [(256, [1]), (16, [15, 16, 17]), (16, [700, 0, 33, 129, 512]), (64, [128 + i for i in range(17)]), (32, [40 * i for i in range(37)])])
def test_against_the_oracle(ops, hq, hkv, bs, lens):
    nblk = sum(-(-c // bs) for c in lens) + 1
    kv, ks, vs = bind_random_cache(ops, 1, nblk, hkv, bs, seed=21)
    tables, q = make_tables(lens, bs, nblk, seed=22), bf(len(lens), hq, 128, seed=23)
    ctx = torch.tensor(lens, dtype=torch.int32)
    want = paged_decode_ref(q, ks[0], vs[0], ctx, tables, 0.09)
    for page in range(nblk):                          # whatever no context covers holds NaN
        live = torch.zeros(bs, dtype=torch.bool)
        for i, c in enumerate(lens):
            for w in range(-(-c // bs)):
                if tables[i, w] == page:
                    live[:min(bs, c - w * bs)] = True
        kv[:, 0, page][:, :, ~live.cuda()] = float("nan")
    got = ops.paged_decode(0, q.cuda(), tables.cuda(), ctx.cuda(), 0.09)
    assert_close_bf16(got, want, f"{hq}/{hkv} {bs}")
    for i, c in enumerate(lens):
        assert c > 0 or got[i].abs().max().item() == 0.0


@pytest.mark.parametrize("hq,hkv", [(2, 2), (4, 2)])
@pytest.mark.parametrize("lens", [[1], [16, 17, 1, 0, 300], [33 * i + 1 for i in range(30)]])
def test_fused_form(ops, hq, hkv, lens):
    bs, n = 16, len(lens)
    nblk = sum(-(-c // bs) for c in lens) + 1
    kv, ks, vs = bind_random_cache(ops, 2, nblk, hkv, bs, seed=24)
    tables, row = make_tables(lens, bs, nblk, seed=25), bf(n, (hq + 2 * hkv) * 128, seed=26)
    g = torch.Generator().manual_seed(27)
    qw, kw = (1 + 0.1 * torch.randn(128, generator=g)).to(torch.bfloat16), (1 + 0.1 * torch.randn(128, generator=g)).to(torch.bfloat16)
    table, ctx = rope_table(128, 2048, 1e6), torch.tensor(lens, dtype=torch.int32)
    pos = (ctx.long() - 1).clamp(min=0)
    q = rope_ref(table, pos, rmsnorm_ref(row[:, :hq * 128].view(n, hq, 128), qw, 1e-6))
    k = rope_ref(table, pos, rmsnorm_ref(row[:, hq * 128:(hq + hkv) * 128].view(n, hkv, 128), kw, 1e-6))
    v = row[:, (hq + hkv) * 128:].view(n, hkv, 128)
    for i, c in enumerate(lens):
        if c:
            page, at = tables[i, (c - 1) // bs].item(), (c - 1) % bs
            ks[1][page, at], vs[1][page, at] = k[i], v[i]
    want = paged_decode_ref(q, ks[1], vs[1], ctx, tables, 128 ** -0.5)
    got = ops.paged_decode_fused(1, row.cuda(), hq, qw.cuda(), kw.cuda(), table.cuda(), 1e-6, tables.cuda(), ctx.cuda(), 128 ** -0.5)
    assert_close_bf16(got, want, "fused", rel_l2=6e-3, ulps=3.0)          # its own q and k carry one more bf16 rounding than the oracle's order of operations
    have_k, have_v = to_logical(kv[0, 1].cpu()), to_logical(kv[1, 1].cpu())
    assert torch.equal(have_v, vs[1])
    assert_close_bf16(have_k, ks[1], "appended keys", ulps=1.01)
