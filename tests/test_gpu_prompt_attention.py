"""The persistent prompt-attention kernel (csrc/fa_tc.cuh) at the sizes where its tiling can go wrong: edges of the 64-key blocks and
128-row tiles, head groups that pair heads and groups that pair row blocks, more work items than one CTA's list holds, a scale that is not
positive, results that are only 16-byte aligned, and the scatter in front of it at both of its grid sizes.

Tolerance: as the other bf16 attention tests, two roundings of the result's scale and 4e-3 in relative L2 (P and the result are rounded to
bf16, 2^-9 relative each)."""
import pytest
import torch

from oracle.paged_attention_ref import varlen_prefill_ref
from test_gpu_kernels import assert_close_bf16, bf, bind_random_cache, make_tables

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from nanovllm import ops as _ops
    return _ops


def cu(lens):
    return torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32)


@pytest.mark.parametrize("hq,hkv", [(4, 2), (3, 1), (2, 2), (8, 1)])
@pytest.mark.parametrize("lens", [[63, 64, 65], [127, 128, 129, 1], [255, 256, 257], [640, 2, 383]])
def test_edges_of_blocks_and_tiles(ops, hq, hkv, lens):
    tot = sum(lens)
    q, k, v = bf(tot, hq, 128, seed=1), bf(tot, hkv, 128, seed=2), bf(tot, hkv, 128, seed=3)
    c = cu(lens)
    want = varlen_prefill_ref(q, k, v, c, c, 128 ** -0.5, p_dtype=torch.bfloat16)
    got = ops.paged_prefill(0, q.cuda(), k.cuda(), v.cuda(), c.cuda(), c.cuda(), max(lens), max(lens), 128 ** -0.5)
    assert_close_bf16(got, want, f"{hq}/{hkv} {lens}")


@pytest.mark.parametrize("scale", [-0.05, 0.0])
def test_scale_that_is_not_positive(ops, scale):
    lens = [130, 70]
    q, k, v = bf(200, 4, 128, seed=4), bf(200, 2, 128, seed=5), bf(200, 2, 128, seed=6)
    c = cu(lens)
    want = varlen_prefill_ref(q, k, v, c, c, scale, p_dtype=torch.bfloat16)
    got = ops.paged_prefill(0, q.cuda(), k.cuda(), v.cuda(), c.cuda(), c.cuda(), 130, 130, scale)
    assert_close_bf16(got, want, f"scale {scale}")


def test_more_items_than_a_list_holds(ops):
    """900 sequences x 16 head pairs: over 96 items for each of 148 CTAs, so the grid grows; every sequence must still be written."""
    lens = [1 + i % 3 for i in range(900)]
    tot, hq, hkv = sum(lens), 32, 8
    q, k, v = bf(tot, hq, 128, seed=7), bf(tot, hkv, 128, seed=8), bf(tot, hkv, 128, seed=9)
    c = cu(lens)
    want = varlen_prefill_ref(q, k, v, c, c, 128 ** -0.5, p_dtype=torch.bfloat16)
    got = ops.paged_prefill(0, q.cuda(), k.cuda(), v.cuda(), c.cuda(), c.cuda(), 3, 3, 128 ** -0.5)
    assert_close_bf16(got, want, "900 sequences")


def test_result_rows_of_16_byte_alignment(ops):
    """Rows 8 elements past a 32-byte boundary take the 16-byte stores; nothing is written between them."""
    lens = [100, 33]
    q, k, v = bf(133, 4, 128, seed=10), bf(133, 2, 128, seed=11), bf(133, 2, 128, seed=12)
    c = cu(lens)
    want = varlen_prefill_ref(q, k, v, c, c, 128 ** -0.5, p_dtype=torch.bfloat16)
    buf = torch.full((133, 4 * 128 + 8), 7.0, dtype=torch.bfloat16, device="cuda")
    out = buf.as_strided((133, 4, 128), (4 * 128 + 8, 128, 1), 8)
    ops.paged_prefill(0, q.cuda(), k.cuda(), v.cuda(), c.cuda(), c.cuda(), 100, 100, 128 ** -0.5, out=out)
    assert_close_bf16(out, want, "strided result")
    assert (buf[:, :8] == 7.0).all()


@pytest.mark.parametrize("n,hkv", [(5, 8), (2400, 8), (19000, 1)])
def test_scatter_at_both_grid_sizes(ops, n, hkv):
    bs = 16
    nblk = -(-n // bs) + 1
    kv, _, _ = bind_random_cache(ops, 1, nblk, hkv, bs, seed=13)
    row = bf(n, 2 * hkv * 128 + 8, seed=14).cuda()
    slots = torch.randperm(nblk * bs, generator=torch.Generator().manual_seed(15))[:n].to(torch.int32)
    slots[n // 2] = -1
    want = kv.clone()
    k, v = row[:, :hkv * 128].view(n, hkv, 128), row[:, hkv * 128:2 * hkv * 128].view(n, hkv, 128)
    live = (slots >= 0).cuda()
    blk, at = (slots // bs).long().cuda()[live], (slots % bs).long().cuda()[live]
    want[0, 0][blk, :, at] = k[live]
    want[1, 0][blk, :, at] = v[live]
    ops.store_kv(0, k, v, slots.cuda())
    assert torch.equal(kv, want)


def test_pages_under_a_prefix(ops):
    """Portions whose first query is in the middle of a block, over pages smaller and larger than a block."""
    for bs in (16, 128):
        len_k, len_q = [190, 64, 333], [65, 1, 205]
        nblk = sum(-(-c // bs) for c in len_k) + 1
        kv, ks, vs = bind_random_cache(ops, 1, nblk, 1, bs, seed=16)
        tables = make_tables(len_k, bs, nblk, seed=17)
        q = bf(sum(len_q), 3, 128, seed=18)
        want = varlen_prefill_ref(q, None, None, cu(len_q), cu(len_k), 128 ** -0.5, tables, ks[0], vs[0], p_dtype=torch.bfloat16)
        got = ops.paged_prefill(0, q.cuda(), None, None, cu(len_q).cuda(), cu(len_k).cuda(), max(len_q), max(len_k), 128 ** -0.5,
                                block_tables=tables.cuda(), num_kv_heads=1)
        assert_close_bf16(got, want, f"prefix, pages of {bs}")
