"""Single-token latent attention on tcgen05 (csrc/latent_decode.cu): contexts around the 64-key tiles (and twice them), steps with fewer and more tiles than CTAs,
empty rows, stale cache rows that hold NaN, windows, sinks, both rotation layouts, fewer heads than columns, page sizes on both sides of a tile.

Reference: the general path of the same entry point in fp32 on the same values (held to float64 by test_gpu_tafopel.py).  P is rounded to bf16
(2^-9 relative) and so is the result."""
import pytest
import torch

from test_gpu_kernels import assert_close_bf16, bf, make_tables

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rank,H", [(512, 16), (256, 16), (512, 5)])
@pytest.mark.parametrize("lens,bs,window,layout", [([1], 256, 0, 0), ([127, 128, 129, 0, 400], 16, 0, 1), ([300, 5, 1000], 128, 200, 0), ([3000, 1, 2500], 256, 0, 1),
                                                   ([17 * i + 1 for i in range(200)], 32, 0, 0)])
def test_against_the_general_path(rank, H, lens, bs, window, layout):
    from nanovllm import mixops as mx
    from nanovllm.layers.rotary_embedding import build_banded_cos_sin
    n, rd = len(lens), 64
    nblk = sum(-(-c // bs) for c in lens) + 1
    tables = make_tables(lens, bs, nblk, seed=50)
    cache = bf(nblk * bs, rank + rd, seed=51).cuda()
    q_lat, q_raw = bf(H, n, rank, seed=52).cuda(), bf(n, H, 128 + rd, seed=53).cuda()
    sink = torch.linspace(-1, 1, H).cuda() if layout == 0 else None
    cs = build_banded_cos_sin(rd, 4096, 1e4, None, "cuda")
    spans = mx.StepSpans(n, 1, None, None, torch.tensor(lens, dtype=torch.int32).cuda())
    args = (tables.cuda(), bs, spans, sink, cs, 0.03)
    live = torch.tensor(lens) > 0
    want = mx.latent_attention(q_lat.float(), q_raw.float(), 128, cache.float(), *args, window=window, layout=layout)
    dead = torch.ones(nblk * bs, dtype=torch.bool)
    for i, c in enumerate(lens):
        p = torch.arange(c)
        dead[tables[i][p // bs].long() * bs + p % bs] = False
    cache[dead.cuda()] = float("nan")
    got = mx.latent_attention(q_lat, q_raw, 128, cache, *args, window=window, layout=layout)
    assert_close_bf16(got[:, live.cuda()], want[:, live.cuda()], f"{rank} {H} {bs}", rel_l2=6e-3, ulps=3.0)


@pytest.mark.parametrize("H,rank,rd,bs", [(17, 256, 64, 256), (4, 128, 64, 256), (4, 256, 32, 256), (4, 256, 64, 24)])
def test_other_sizes_take_the_general_form(H, rank, rd, bs):
    from nanovllm import mixops as mx
    from nanovllm.layers.rotary_embedding import build_banded_cos_sin
    lens = [70, 200]
    nblk = sum(-(-c // bs) for c in lens) + 1
    tables, cache = make_tables(lens, bs, nblk, seed=54), bf(nblk * bs, rank + rd, seed=55).cuda()
    q_lat, q_raw = bf(H, 2, rank, seed=56).cuda(), bf(2, H, 128 + rd, seed=57).cuda()
    cs = build_banded_cos_sin(rd, 4096, 1e4, None, "cuda")
    args = (tables.cuda(), bs, mx.StepSpans(2, 1, None, None, torch.tensor(lens, dtype=torch.int32).cuda()), None, cs, 0.03)
    want = mx.latent_attention(q_lat.float(), q_raw.float(), 128, cache.float(), *args)
    assert_close_bf16(mx.latent_attention(q_lat, q_raw, 128, cache, *args), want, "general form", rel_l2=6e-3, ulps=3.0)


@pytest.mark.parametrize("n", [1, 200])
def test_lengths_written_by_the_kernel_in_front(n):
    """The lengths come out of this library's own gather of rows, whose launch lets the next one begin before it has written them."""
    from nanovllm import mixops as mx, ops
    from nanovllm.layers.rotary_embedding import build_banded_cos_sin
    rank, rd, H, bs, most = 256, 64, 4, 128, 2048
    tables = torch.arange(n * most // bs, dtype=torch.int32).view(n, -1).cuda()
    cache, q_lat, q_raw = bf(most * n, rank + rd, seed=58).cuda(), bf(H, n, rank, seed=59).cuda(), bf(n, H, rd, seed=60).cuda()
    cs = build_banded_cos_sin(rd, most, 1e4, None, "cuda")
    g = torch.Generator().manual_seed(61)
    rows = 1 << 18                                                       # the step's lengths are the last of many rows: they are written late
    for turn in range(3):
        lens = torch.randint(1, most, (n,), generator=g, dtype=torch.int32).cuda()
        held = torch.zeros(rows * 8 + (n + 7) // 8 * 8, dtype=torch.int32, device="cuda")
        source = torch.zeros_like(held)
        source[rows * 8:rows * 8 + n] = lens
        ids = torch.arange(held.numel() // 8, device="cuda")
        spans = lambda t: mx.StepSpans(n, 1, None, None, t)
        want = mx.latent_attention(q_lat, q_raw, 0, cache, tables, bs, spans(lens), None, cs, 0.03)
        torch.cuda.synchronize()
        ops.embedding(ids, source.view(torch.bfloat16).view(-1, 16), out=held.view(torch.bfloat16).view(-1, 16))
        got = mx.latent_attention(q_lat, q_raw, 0, cache, tables, bs, spans(held[rows * 8:rows * 8 + n]), None, cs, 0.03)
        assert torch.equal(got, want)


def test_pages_below_the_window_may_be_absent():
    from nanovllm import mixops as mx
    from nanovllm.layers.rotary_embedding import build_banded_cos_sin
    H, rank, rd, bs, window, lens = 4, 256, 64, 16, 100, [700, 391, 60]
    nblk = sum(-(-c // bs) for c in lens)
    cache = bf((nblk + 1) * bs, rank + rd, seed=62).cuda()
    cache[:bs] = float("nan")
    tables = make_tables(lens, bs, nblk, seed=63)
    tables[tables >= 0] += 1
    q_lat, q_raw = bf(H, 3, rank, seed=64).cuda(), bf(3, H, rd, seed=65).cuda()
    cs = build_banded_cos_sin(rd, 1024, 1e4, None, "cuda")
    spans = mx.StepSpans(3, 1, None, None, torch.tensor(lens, dtype=torch.int32).cuda())
    call = lambda t: mx.latent_attention(q_lat, q_raw, 0, cache, t.cuda(), bs, spans, None, cs, 0.03, window=window)
    want = call(tables)
    for i, l in enumerate(lens):
        tables[i, :max(l - window, 0) // bs] = -1
    assert torch.equal(call(tables), want) and torch.isfinite(want).all()


@pytest.mark.parametrize("rank,bs", [(512, 8), (512, 64), (256, 16), (512, 384)])
def test_tile_edges_and_a_maximum_that_moves(rank, bs):
    """Contexts around the 64-key tiles and over several turns of the rings; keys that grow with their position, so that the reference maximum moves in tile after tile.
    Only the latents grow: the kernel has the rotated query in bf16, 2^-9 of it off, which times a rotated key 35 times as long (0.03 * 35 * sqrt(64) * 2^-9 = 0.016 of a score)
    would show as 1.6 % of the weights."""
    from nanovllm import mixops as mx
    from nanovllm.layers.rotary_embedding import build_banded_cos_sin
    H, rd, lens = 16, 64, [63, 64, 65, 127, 1, 705, 1409, 192]
    n, nblk = len(lens), sum(-(-c // bs) for c in lens) + 1
    tables, cache = make_tables(lens, bs, nblk, seed=70), bf(nblk * bs, rank + rd, seed=71)
    for i, c in enumerate(lens):
        p = torch.arange(c)
        rows = tables[i][p // bs].long() * bs + p % bs
        cache[rows, :rank] = (cache[rows, :rank].float() * (0.05 + p[:, None] / 40)).bfloat16()
    q_lat, q_raw = bf(H, n, rank, seed=72).cuda(), bf(n, H, 128 + rd, seed=73).cuda()
    cs = build_banded_cos_sin(rd, 4096, 1e4, None, "cuda")
    args = (tables.cuda(), bs, mx.StepSpans(n, 1, None, None, torch.tensor(lens, dtype=torch.int32).cuda()), torch.linspace(-1, 1, H).cuda(), cs, 0.03)
    want = mx.latent_attention(q_lat.float(), q_raw.float(), 128, cache.cuda().float(), *args)
    assert_close_bf16(mx.latent_attention(q_lat, q_raw, 128, cache.cuda(), *args), want, f"{rank} {bs}", rel_l2=6e-3, ulps=3.0)


@pytest.mark.parametrize("rank", [256, 512])
@pytest.mark.parametrize("n,lo,hi,scale,window", [(1, 200, 200, 0.03, 0), (1, 8000, 8000, 0.03, 0), (8, 500, 4000, 0.12, 0), (64, 2048, 4096, 0.03, 0), (64, 2048, 4096, 0.03, 500), (128, 32, 300, 0.03, 0)])
def test_nearest_bf16_but_for_a_few(rank, n, lo, hi, scale, window):
    """Results against float64 on the kernel's own inputs (the query's rotated part in bf16): what is left is the rounding of the result, 2^-9 of a number at most and 0.42 of that in the
    norm, and weights in two bf16 terms (2^-17), which put a result on the other side of a rounding border once in some hundred (measured: 0.0024 of them at most, and 0.0027 with tiles
    of 128 keys)."""
    from nanovllm import mixops as mx
    from nanovllm.layers.rotary_embedding import build_interleaved_cos_sin
    H, rd, d, bs = 16, 64, 128, 64
    lens = [int(lo + (hi - lo) * (i + 0.5) / n) for i in range(n)]
    nblk = sum(-(-c // bs) for c in lens)
    tables = make_tables(lens, bs, nblk, seed=80)
    cache, q_lat, q_raw = bf(nblk * bs, rank + rd, seed=81).cuda(), bf(H, n, rank, seed=82).cuda(), bf(n, H, d + rd, seed=83).cuda()
    cs, sink = build_interleaved_cos_sin(rd, 8192, 1e4, None, "cuda"), torch.linspace(-1, 1, H).cuda()
    got = mx.latent_attention(q_lat, q_raw, d, cache, tables.cuda(), bs, mx.StepSpans(n, 1, None, None, torch.tensor(lens, dtype=torch.int32).cuda()), sink, cs, scale, window=window)
    off = size = moved = 0.0
    for i, c in enumerate(lens):
        p = torch.arange(max(0, c - window) if window else 0, c)
        kv = cache[(tables[i][p // bs].long() * bs + p % bs).cuda()].double()
        u, w, cos, sin = q_raw[i, :, d::2].float(), q_raw[i, :, d + 1::2].float(), cs[c - 1, :rd // 2], cs[c - 1, rd // 2:]
        rot = torch.stack((u * cos - w * sin, w * cos + u * sin), -1).flatten(1).bfloat16()
        s = torch.cat((torch.cat((q_lat[:, i], rot), 1).double() @ kv.t() * scale, sink[:, None].double()), 1)
        want = torch.softmax(s, 1)[:, :-1] @ kv[:, :rank]
        off, size, moved = off + (got[:, i].double() - want).square().sum().item(), size + want.square().sum().item(), moved + (got[:, i] != want.bfloat16()).sum().item()
    assert (off / size) ** 0.5 < 2.0 ** -9 and moved < 0.01 * got.numel()
