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


# ---- the same kernel over token-major cache rows (windowed attention) and over formed keys and values (latent attention) --------------------
@pytest.fixture(scope="module")
def mx():
    from nanovllm import mixops as _mx
    return _mx


def paged_rows(len_k, bs, cols, seed):
    nblk = sum(-(-c // bs) for c in len_k) + 1
    tables = make_tables(len_k, bs, nblk, seed=seed)
    return bf(nblk * bs, cols, seed=seed + 1).cuda(), tables.cuda()


def spans_of(mx, len_q, len_k):
    return mx.StepSpans(len(len_q), max(len_q), cu(len_q).cuda(), cu(len_k).cuda(), None)


WINDOW_FORMS = {
    "bias and window": dict(slopes=True, window=100),
    "bias alone": dict(slopes=True),
    "window below a block": dict(window=7),
    "chunks and sinks": dict(chunk=96, sinks=True),
    "head gate": dict(gate="heads", out_scale=0.5),
    "element gate, fp32 result": dict(gate="elems", out_f32=True, window=64),
    "negative scale": dict(scale=-0.06),
}


@pytest.mark.parametrize("form", WINDOW_FORMS)
@pytest.mark.parametrize("heads,kv_heads,bs", [(4, 2, 256), (3, 1, 16), (2, 2, 64), (4, 1, 24)])        # pages of 24: the route falls through
def test_windowed_prompts_against_the_fp32_pipe(mx, form, heads, kv_heads, bs):
    """Against the general fp32 path of the same entry point on the same bf16 inputs (test_gpu_tipetar.py and others hold that one to float64): P and
    the result are rounded to bf16, 2^-9 relative each."""
    f = dict(WINDOW_FORMS[form])
    len_q, len_k = [1, 130, 63, 200], [150, 130, 191, 329]
    n, H = sum(len_q), heads
    cache, tables = paged_rows(len_k, bs, kv_heads * 256, 30)
    q = bf(n, H * 128 + 16, seed=31).cuda()
    gate = None
    if f.get("gate"):
        gate = bf(n, (H if f["gate"] == "heads" else H * 128) + 8, seed=32).cuda()[:, :H if f["gate"] == "heads" else H * 128]
    kw = dict(slopes=torch.exp2(-torch.arange(1, H + 1, dtype=torch.float32)).cuda() if f.get("slopes") else None, window=f.get("window", 0), chunk=f.get("chunk", 0),
              sinks=torch.linspace(-1, 2, H).cuda() if f.get("sinks") else None, gate=gate, out_scale=f.get("out_scale", 1.0), out_f32=f.get("out_f32", False))
    args = (q, cache, tables, bs, spans_of(mx, len_q, len_k), H, kv_heads, 128, 128, f.get("scale", 128 ** -0.5))
    got, want = mx.window_attention(*args, **kw), mx.window_attention(*args, fma=True, **kw)
    assert got.dtype == want.dtype
    assert_close_bf16(got, want, form)


@pytest.mark.parametrize("layout", [0, 1])
@pytest.mark.parametrize("len_q,len_k,window,bs", [([64, 129, 1], [64, 129, 300], 0, 256), ([255, 257], [600, 257], 0, 16), ([40, 200], [333, 200], 50, 256)])
def test_latent_prompts_against_attention_over_the_latents(mx, layout, len_q, len_k, window, bs):
    """Keys and values formed per head against the products with the latents themselves, fp32 throughout (the general path on the same values): what
    differs are the bf16 roundings of keys, values and P on one side, 2^-9 relative each, none on the other."""
    from nanovllm.layers.rotary_embedding import build_banded_cos_sin
    H, d, rd, R, n = 4, 128, 64, 64, sum(len_q)
    cache, tables = paged_rows(len_k, bs, R + rd, 40)
    q = bf(n, H, d + rd, seed=41).cuda()
    w = bf(H * (d + 128), R, scale=R ** -0.5, seed=42).cuda()
    sink = torch.linspace(-1, 1, H).cuda() if window == 0 else None
    cs = build_banded_cos_sin(rd, 1024, 1e4, None, "cuda")
    pos = torch.cat([torch.arange(b - a, b) for a, b in zip(len_q, len_k)]).cuda()
    spans = spans_of(mx, len_q, len_k)
    assert mx.latent_expands(q, d, rd, 128, R, 192 ** -0.5, cache, tables, bs, spans)
    assert not mx.latent_expands(q, d, rd, 64, R, 192 ** -0.5, cache, tables, bs, spans)
    uk, uv = w[:H * d].view(H, d, R).float(), w[H * d:].view(H, 128, R).float()
    q_lat = torch.bmm(q[:, :, :d].transpose(0, 1).float(), uk)
    o_lat = mx.latent_attention(q_lat, q.float(), d, cache.float(), tables, bs, spans, sink, cs, 192 ** -0.5, window=window, layout=layout)
    want = torch.bmm(o_lat, uv.transpose(1, 2)).transpose(0, 1).reshape(n, H * 128)
    got = mx.latent_prompt(q, w, d, 128, cache, tables, bs, spans, sink, cs, pos, 192 ** -0.5, window=window, layout=layout)
    assert_close_bf16(got, want, "latent prompts", rel_l2=8e-3, ulps=3.0)


@pytest.mark.parametrize("dims,off", [(64, 128), (16, 128), (6, 128), (64, 124)])
@pytest.mark.parametrize("layout", [0, 1])
def test_rotation_in_place(mx, dims, off, layout):
    """Wide and pair-by-pair accesses (odd sizes, 8-byte aligned starts) against float64; nothing beside the rotated columns changes."""
    from nanovllm.layers.rotary_embedding import build_banded_cos_sin
    n, H = 37, 3
    q = bf(n, H, 192, seed=60).cuda()
    want = q.double()
    pos = torch.arange(n).flip(0).cuda() * 7
    cs = build_banded_cos_sin(dims, 512, 1e4, None, "cuda")
    c, s = cs[pos, :dims // 2].double()[:, None], cs[pos, dims // 2:].double()[:, None]
    lo = slice(off, off + dims, 2) if layout == 0 else slice(off, off + dims // 2)
    hi = slice(off + 1, off + dims, 2) if layout == 0 else slice(off + dims // 2, off + dims)
    u, v = want[..., lo].clone(), want[..., hi].clone()
    want[..., lo], want[..., hi] = u * c - v * s, v * c + u * s
    mx._call("b200m_latent_rotate", q.data_ptr() + 2 * off, q.stride(0), q.stride(1), cs.data_ptr(), dims, pos.data_ptr(), n, H, layout, mx._stream())
    assert (q.double() - want).abs().max().item() <= 2 ** -8 * want.abs().max().item()
    keep = torch.ones(192, dtype=torch.bool)
    keep[off:off + dims] = False
    assert torch.equal(q[..., keep.cuda()].double(), want[..., keep.cuda()])


@pytest.mark.parametrize("bs,window", [(16, 100), (32, 7)])
def test_pages_below_the_window_may_be_absent(mx, bs, window):
    """Table entries of pages that no query sees are -1 and whatever page 0 holds (NaN here) stays out: bit for bit the result with all pages there."""
    heads, kv_heads, len_q, len_k = 4, 2, [40, 130], [700, 391]
    nblk = sum(-(-c // bs) for c in len_k)
    cache = bf((nblk + 1) * bs, kv_heads * 256, seed=70).cuda()
    cache[:bs] = float("nan")
    tables = make_tables(len_k, bs, nblk, seed=71)
    tables[tables >= 0] += 1                                             # page 0 belongs to nobody
    q = bf(sum(len_q), heads * 128, seed=72).cuda()
    call = lambda t: mx.window_attention(q, cache, t.cuda(), bs, spans_of(mx, len_q, len_k), heads, kv_heads, 128, 128, 128 ** -0.5, window=window)
    want = call(tables)
    assert torch.isfinite(want).all()
    for i, (n, l) in enumerate(zip(len_q, len_k)):
        tables[i, :(l - n - window + 1) // bs] = -1
    assert torch.equal(call(tables), want)


def latent_case(mx, H, R, len_q, len_k, bs, seed, known=True):
    from nanovllm.layers.rotary_embedding import build_banded_cos_sin
    n = sum(len_q)
    cache, tables = paged_rows(len_k, bs, R + 64, seed)
    q, w = bf(n, H, 192, seed=seed + 2).cuda(), bf(H * 256, R, scale=R ** -0.5, seed=seed + 3).cuda()
    cs = build_banded_cos_sin(64, max(len_k), 1e4, None, "cuda")
    pos = torch.cat([torch.arange(b - a, b) for a, b in zip(len_q, len_k)]).cuda()
    extra = (max(len_k), sum(len_k)) if known else ()
    spans = mx.StepSpans(len(len_q), max(len_q), cu(len_q).cuda(), cu(len_k).cuda(), None, *extra)
    return q, w, cache, tables, spans, cs, pos


def over_the_latents(mx, case, bs, sink, window):
    q, w, cache, tables, spans, cs, pos = case
    n, H = q.shape[:2]
    R = w.shape[1]
    uk, uv = w[:H * 128].view(H, 128, R).float(), w[H * 128:].view(H, 128, R).float()
    o = mx.latent_attention(torch.bmm(q[:, :, :128].transpose(0, 1).float(), uk), q.float(), 128, cache.float(), tables, bs, spans, sink, cs, 192 ** -0.5, window=window)
    return torch.bmm(o, uv.transpose(1, 2)).transpose(0, 1).reshape(n, H * 128)


@pytest.mark.parametrize("window", [0, 90])
@pytest.mark.parametrize("known", [True, False])
@pytest.mark.parametrize("group", [1, 2, 3, 4])
def test_latent_prompts_of_ragged_steps(mx, window, known, group, monkeypatch):
    """Sequences of very different lengths, with and without lengths on the host, a window that cuts most keys, and keys and values formed for a few heads at a
    time: as attention over the latents."""
    H, R, len_q, len_k, bs = 4, 64, [64, 1, 129, 30], [1200, 5, 129, 700], 16
    case = latent_case(mx, H, R, len_q, len_k, bs, 80, known)
    q, w, cache, tables, spans, cs, pos = case
    total, most = mx._latent_rows(q.shape[0], tables, bs, spans, window)
    seen = [min(k, a + window - 1) if window else k for a, k in zip(len_q, len_k)]
    assert sum(seen) <= total and max(seen) <= most
    if known and not window:
        assert (total, most) == (sum(len_k), max(len_k))
    sink = torch.linspace(-1, 1, H).cuda()
    want = over_the_latents(mx, case, bs, sink, window)
    monkeypatch.setattr(mx, "LATENT_KV_BYTES", total * 512 * group)
    got = mx.latent_prompt(q, w, 128, 128, cache, tables, bs, spans, sink, cs, pos, 192 ** -0.5, window=window)
    assert_close_bf16(got, want, "ragged", rel_l2=8e-3, ulps=3.0)


@pytest.mark.parametrize("len_q,len_k,window,rows", [([100] * 31 + [4096], [100] * 31 + [4096], 0, 31 * 100 + 4096), ([16, 16], [30000, 12000], 1024, 2 * 1039)])
def test_latent_prompts_hold_the_rows_that_are_seen(mx, len_q, len_k, window, rows):
    """A long sequence beside short ones, and a short portion behind a long context under a window: memory for the real rows alone."""
    H, R, bs = 4, 64, 256
    q, w, cache, tables, spans, cs, pos = latent_case(mx, H, R, len_q, len_k, bs, 85)
    args = (q, w, 128, 128, cache, tables, bs, spans, None, cs, pos, 192 ** -0.5)
    assert mx.latent_expands(q, 128, 64, 128, R, 192 ** -0.5, cache, tables, bs, spans, window)
    mx.latent_prompt(*args, window=window)
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    held = torch.cuda.memory_allocated()
    out = mx.latent_prompt(*args, window=window)
    used = torch.cuda.max_memory_allocated() - held - out.numel() * 2
    spare = 3 << 20                                                      # the allocator hands out a larger free block when less than 1 MiB of it would be left
    assert used <= rows * (H * 512 + (R + 64) * 2) + spare               # the padded rows would be 302 and 138 MB
    assert used <= mx.latent_scratch_bytes(H, 128, 128, R + 64, rows) + spare


def test_rows_seen_through_a_window(mx):
    """The prefix over sequences, at sizes around the block of 1024 that forms it; sequences without queries count nothing."""
    for S in (1, 31, 1024, 1025, 2500):
        g = torch.Generator().manual_seed(S)
        q = torch.randint(0, 50, (S,), generator=g)
        k = q + torch.randint(0, 300, (S,), generator=g)
        out = torch.empty(S + 1, dtype=torch.int32, device="cuda")
        a, b = cu(q.tolist()).cuda(), cu(k.tolist()).cuda()
        for window in (1, 64, 2 ** 31 - 1):
            mx._call("b200m_latent_visible", a.data_ptr(), b.data_ptr(), S, window, out.data_ptr(), mx._stream())
            want = torch.where(q > 0, torch.minimum(k, q + window - 1), torch.zeros_like(q))
            assert torch.equal(out.cpu(), cu(want.tolist()))
