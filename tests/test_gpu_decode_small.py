"""Paged decode of small steps (csrc/decode_small.cu): one CTA and clusters of 2, 4 and 8 per context (the library says which: a step that falls
to the other kernels fails the tests that name a form), every head group, contexts around chunk and page edges, empty rows, stale rows, and the fused
form's append.  Tolerance as the other decode tests; the forms are those of a device with 148 SMs."""
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
    fused(ops, hq, hkv, lens)


def fused(ops, hq, hkv, lens):
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


def splits(ops, batch, hq, width):
    h = ops.nat.handle()
    return h.lib.b200_decode_small_splits(h.ptr, batch, hq, width)


def decode(ops, hq, hkv, bs, lens, width, splits_here, seed):
    nblk = sum(-(-c // bs) for c in lens) + 1
    kv, ks, vs = bind_random_cache(ops, 1, nblk, hkv, bs, seed=seed)
    tables, q = make_tables(lens, bs, nblk, seed=seed + 1), bf(len(lens), hq, 128, seed=seed + 2)
    tables = torch.cat((tables, torch.full((len(lens), max(0, width - tables.shape[1])), -1, dtype=torch.int32)), 1)
    assert splits(ops, len(lens), hq, tables.shape[1]) == splits_here
    ctx = torch.tensor(lens, dtype=torch.int32)
    got = ops.paged_decode(0, q.cuda(), tables.cuda(), ctx.cuda(), 0.09)
    assert_close_bf16(got, paged_decode_ref(q, ks[0], vs[0], ctx, tables, 0.09), f"{hq}/{hkv} {bs}")


@pytest.mark.parametrize("hq,hkv,rows", [(8, 8, 18), (16, 8, 12), (32, 8, 18), (64, 8, 9), (16, 2, 37), (2, 2, 74)])
def test_a_cta_per_context(ops, hq, hkv, rows):
    """More than half of the SMs have a (sequence, kv head): no cluster, the result leaves from the first meeting."""
    decode(ops, hq, hkv, 16, [(37 * i) % 301 for i in range(rows)], 0, 1, 31)


@pytest.mark.parametrize("hq,hkv,rows,tokens,splits_here", [(4, 2, 1, 16384, 8), (4, 2, 16, 8192, 4), (4, 2, 37, 4096, 2), (16, 8, 18, 2048, 1), (16, 2, 37, 512, 1)])
def test_longest_context_of_each_form(ops, hq, hkv, rows, tokens, splits_here):
    """At the widest table the rule takes, full contexts beside short ones; a page more is a step for the other kernels."""
    decode(ops, hq, hkv, 256, [tokens, 1, 17, 0][:rows] + [5] * (rows - 4), tokens // 256, splits_here, 34)
    assert splits(ops, rows, hq, tokens // 256 + 1) == 0


@pytest.mark.parametrize("hq,hkv,lens,splits_here", [(16, 8, [25 * i for i in range(18)], 1), (8, 8, [25 * i + 1 for i in range(10)], 1)])
def test_fused_form_of_a_cta_per_context(ops, hq, hkv, lens, splits_here):
    ops.bind_kv_cache(torch.zeros(ops.kv_cache_shape(2, 4, hkv, 16, 128), dtype=torch.bfloat16, device="cuda"))
    assert splits(ops, len(lens), hq, -(-max(lens) // 16)) == splits_here
    fused(ops, hq, hkv, lens)
