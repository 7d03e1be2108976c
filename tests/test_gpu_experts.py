"""The grouped expert GEMMs on tcgen05 (csrc/moe_tc.cu) at the sizes where their tiling can go wrong: experts with no rows, one, a tile less
one, a tile, a tile and one, odd numbers of tiles; K that is no multiple of a stage; one and several blocks of weight rows; both forms, every
activation and result type, gathered rows with and without weights.

Reference: the same bf16 operands multiplied in fp32 by torch.  Both sides accumulate in fp32 in another order (1e-5 relative); bf16 results
carry one more rounding (2^-9)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mx():
    from nanovllm import mixops as _mx
    return _mx


def routing(counts, top, seed):
    """idx [n, top] in which expert e is chosen counts[e] times, in a shuffled order (-1 fills up)."""
    g = torch.Generator().manual_seed(seed)
    flat = torch.cat([torch.full((c,), e) for e, c in enumerate(counts)])
    flat = torch.cat([flat, torch.full((-flat.numel() % top,), -1)])
    return flat[torch.randperm(flat.numel(), generator=g)].view(-1, top).to(torch.int32).cuda()


COUNTS = {"few": [0, 1, 5, 63, 64, 0, 2], "edges": [65, 128, 0, 129, 127, 1, 192], "many": [700, 64, 257], "one expert": [0, 0, 333]}


@pytest.mark.parametrize("counts", COUNTS)
@pytest.mark.parametrize("act,gather,weighted,out_f32", [(0, False, False, True), (1, True, True, False), (2, True, False, False), (2, True, True, True)])
@pytest.mark.parametrize("N,K", [(256, 64), (512, 200), (768, 1024)])
@pytest.mark.parametrize("form", ["stream", "rows"])
def test_grouped_gemm(mx, counts, act, gather, weighted, out_f32, N, K, form, monkeypatch):
    counts, top = COUNTS[counts], 3
    E = len(counts)
    idx = routing(counts, top, 1)
    n = idx.shape[0]
    g = torch.Generator(device="cuda").manual_seed(2)
    rows, pos_of, tile_expert, num_tiles = mx.moe_align(idx, E)
    cap = rows.numel()
    A = torch.randn(n if gather else cap, K + 8, generator=g, device="cuda").to(torch.bfloat16)[:, :K]
    W = (torch.randn(E, N, K, generator=g, device="cuda") * K ** -0.5).to(torch.bfloat16)
    wgt = torch.rand(n, top, generator=g, device="cuda") if weighted else None
    if not gather:
        A = A.clone()
        A[rows < 0] = float("nan")                   # padding rows of the grouped buffer hold anything: nothing may come of them
    lib = mx.nat.load_mix()
    real = lib.b200m_moe_gemm
    hint = 1 if form == "stream" else 1 << 20

    class Lib:
        def __getattr__(self, name):
            if name != "b200m_moe_gemm":
                return getattr(lib, name)
            return lambda *a: real(*a[:-3], (a[-3] & 255) | hint << 8, *a[-2:])

    monkeypatch.setattr(mx.nat, "load_mix", lambda: Lib())
    got = mx.moe_gemm(A, rows, tile_expert, num_tiles, W, wgt=wgt, top=top, act=act, out_f32=out_f32, gather=gather)
    live = (rows >= 0).nonzero().view(-1)
    pair = rows[live].long()
    e = idx.view(-1)[pair].long()
    x = A[pair // top].float() if gather else A[live].float()
    if weighted:
        x = (x * wgt.view(-1)[pair, None]).to(torch.bfloat16).float()       # the expert's input is a bf16 tensor
    y = torch.empty(live.numel(), N, device="cuda")
    for k in range(E):
        y[e == k] = x[e == k] @ W[k].float().T
    if act == 1:
        y = torch.relu(y).square()
    elif act == 2:
        y = torch.nn.functional.silu(y[:, :N // 2]) * y[:, N // 2:]
    have = got[live].float()
    assert torch.isfinite(have).all()
    err = ((have - y).norm() / y.norm()).item()
    assert err < (2e-5 if out_f32 else 4e-3), err
    assert (have - y).abs().max().item() <= (1e-4 if out_f32 else 2 ** -7) * max(1.0, y.abs().max().item())


@pytest.mark.parametrize("n,E,top", [(1, 5, 2), (300, 40, 3), (3000, 7, 4), (700, 1500, 2)])
def test_grouping(mx, n, E, top):
    """Every pair lands in its expert's run once, runs start on tiles, the rest is padding; one CTA, clusters, and more experts than counters."""
    g = torch.Generator().manual_seed(3)
    idx = torch.randint(-1, E, (n, top), generator=g).to(torch.int32)
    if E == 7:
        idx[idx == 2] = 5                            # an expert without rows, one with most
    rows, pos_of, tile_expert, num_tiles = (t.cpu() for t in mx.moe_align(idx.cuda(), E))
    flat, used = idx.view(-1), int(num_tiles)
    assert torch.equal(pos_of < 0, flat < 0)
    live = (flat >= 0).nonzero().view(-1)
    assert torch.equal(rows[pos_of[live].long()], live.to(torch.int32))
    assert int((rows >= 0).sum()) == live.numel() and bool((rows[used * 64:] < 0).all())
    assert torch.equal(tile_expert[pos_of[live].long() // 64], flat[live])
    counts = torch.bincount(flat[live].long(), minlength=E)
    assert used == int(((counts + 63) // 64).sum()) and torch.equal(torch.bincount(tile_expert[:used].long(), minlength=E), (counts + 63) // 64)


@pytest.mark.parametrize("n", [1, 200, 2600])
@pytest.mark.parametrize("act,N,weigh_inputs,shared,ident", [(1, 256, True, True, False), (2, 512, False, True, True), (2, 192, False, False, True)])
def test_one_call_against_its_parts(mx, n, act, N, weigh_inputs, shared, ident):
    """The one-call form against the single entry points on the same inputs: the same operations, so only the order of fp32 sums may differ."""
    E, top, K, width = 9, 3, 136, 260 if N == 192 else 512
    g = torch.Generator(device="cuda").manual_seed(4)
    rn = lambda *s: torch.randn(*s, generator=g, device="cuda")
    idx = torch.randint(-1 if ident else 0, E, (n, top), generator=g, device="cuda").to(torch.int32)
    wgt, h = torch.rand(n, top, generator=g, device="cuda"), rn(n, K).to(torch.bfloat16)
    w_in, w_out = (rn(E, N, K) * K ** -0.5).to(torch.bfloat16), (rn(E, width, N // act) * 0.1).to(torch.bfloat16)
    sh, gate = (rn(n, width).to(torch.bfloat16), rn(n, 3)[:, 1]) if shared else (None, None)
    x = rn(n, width) if ident else None
    got = mx.moe_experts(h, idx, wgt, w_in, w_out, act, weigh_inputs, sh, gate, x)
    rows, pos_of, tile_expert, num_tiles = mx.moe_align(idx, E)
    inter = mx.moe_gemm(h, rows, tile_expert, num_tiles, w_in, wgt=wgt if weigh_inputs else None, top=top, act=act, gather=True)
    res = mx.moe_gemm(inter, rows, tile_expert, num_tiles, w_out, out_f32=True)
    want = mx.moe_combine(res, pos_of, top, n, sh, gate, wgt=None if weigh_inputs else wgt, ident=x)
    assert ((got - want).norm() / want.norm()).item() < 1e-5


@pytest.mark.parametrize("N", [512, 640])
def test_one_call_counts_as_its_steps_do(mx, N):
    """The launches of the one call are those of grouping, copy (where the first GEMM reads grouped rows), GEMMs and sum called one by one, with the same result; the
    fp32 rows are no part of its workspace."""
    from nanovllm import ops
    n, top, E, width = 3000, 4, 16, 512
    idx = routing([n * top // E] * E, top, 5)
    g = torch.Generator(device="cuda").manual_seed(6)
    A = torch.randn(n, width, generator=g, device="cuda").to(torch.bfloat16)
    w_in = (torch.randn(E, N, width, generator=g, device="cuda") * width ** -0.5).to(torch.bfloat16)
    w_out = (torch.randn(E, width, N // 2, generator=g, device="cuda") * width ** -0.5).to(torch.bfloat16)
    wgt = torch.rand(n, top, generator=g, device="cuda")
    at = [ops.LAUNCHES[0]]
    got = mx.moe_experts(A, idx, wgt, w_in, w_out, 2, False)
    at.append(ops.LAUNCHES[0])
    rows, pos_of, tile_expert, num_tiles = mx.moe_align(idx, E)
    inter = mx.moe_gemm(A, rows, tile_expert, num_tiles, w_in, top=top, act=2, gather=True)
    want = mx.moe_combine(mx.moe_gemm(inter, rows, tile_expert, num_tiles, w_out, out_f32=True), pos_of, top, n, None, None, wgt=wgt)
    at.append(ops.LAUNCHES[0])
    assert at[1] - at[0] == at[2] - at[1] == (5 if N % 256 == 0 else 4)
    assert (got - want).norm() <= 2e-5 * want.norm()
    cap = mx.moe_capacity(n * top, E)
    assert mx.nat.load_mix().b200m_moe_experts_workspace_bytes(n * top, E, width, N // 2) <= cap * 2 * (width + N // 2) + 12 * cap + 4096


@pytest.mark.parametrize("act,N,K,width", [(1, 256, 64, 2048), (2, 2048, 64, 1024), (2, 512, 200, 2048), (1, 768, 264, 2176)])
@pytest.mark.parametrize("n", [3, 160])
def test_few_rows_over_several_turns(mx, n, act, N, K, width):
    """One call for a few rows of many experts: more items than CTAs at a time, fewer steps of k than the ring has stages, tiles that end the grid's last turn anywhere; in turn with calls
    of other routings, whose kernels begin while those of the call before are under way."""
    E, top = 40, 2
    g = torch.Generator(device="cuda").manual_seed(n + N)
    inter = N // act
    w_in = (torch.randn(E, N, K, generator=g, device="cuda") * K ** -0.5).to(torch.bfloat16)
    w_out = (torch.randn(E, width, inter, generator=g, device="cuda") * inter ** -0.5).to(torch.bfloat16)
    calls = []
    for turn in range(3):
        idx = torch.stack([torch.randperm(E, generator=g, device="cuda")[:top] for _ in range(n)]).to(torch.int32)
        h, wgt = torch.randn(n, K, generator=g, device="cuda").to(torch.bfloat16), torch.rand(n, top, generator=g, device="cuda")
        calls.append((h, idx, wgt))
    torch.cuda.synchronize()
    got = [mx.moe_experts(h, idx, wgt, w_in, w_out, act, False) for h, idx, wgt in calls]
    for (h, idx, wgt), y in zip(calls, got):
        want = torch.zeros(n, width, device="cuda")
        for k in range(top):
            e = idx[:, k].long()
            x = torch.einsum("tk,tnk->tn", h.float(), w_in[e].float())
            x = torch.relu(x).square() if act == 1 else torch.nn.functional.silu(x[:, :inter]) * x[:, inter:]
            want += wgt[:, k, None] * torch.einsum("ti,twi->tw", x.to(torch.bfloat16).float(), w_out[e].float())
        # the activation is rounded to bf16 on both sides, of sums in another order: a few of its values differ by 2^-8
        assert ((y - want).norm() / want.norm()).item() < 1e-3


@pytest.mark.parametrize("act,N,K,width", [(1, 256, 64, 2048), (2, 2048, 64, 1024)])
@pytest.mark.parametrize("n", [1, 64])
def test_steps_whose_choices_are_all_identity_experts(mx, n, act, N, K, width):
    """Without a row for any expert the products' CTAs have no item and leave at once, behind the kernel in front all the same: such steps in turn with ordinary ones, whose
    workspace the allocator takes from the one just given back."""
    E, top = 40, 2
    g = torch.Generator(device="cuda").manual_seed(n + N)
    inter = N // act
    w_in = (torch.randn(E, N, K, generator=g, device="cuda") * K ** -0.5).to(torch.bfloat16)
    w_out = (torch.randn(E, width, inter, generator=g, device="cuda") * inter ** -0.5).to(torch.bfloat16)
    h, wgt = torch.randn(n, K, generator=g, device="cuda").to(torch.bfloat16), torch.rand(n, top, generator=g, device="cuda")
    idx = torch.stack([torch.randperm(E, generator=g, device="cuda")[:top] for _ in range(n)]).to(torch.int32)
    none = torch.full_like(idx, -1)
    want = mx.moe_experts(h, idx, wgt, w_in, w_out, act, False)
    torch.cuda.synchronize()
    for _ in range(4):
        got = [mx.moe_experts(h, i, wgt, w_in, w_out, act, False) for i in (none, idx, none, none, idx)]
        for y, i in zip(got, (none, idx, none, none, idx)):
            assert torch.equal(y, want) if i is idx else not y.any()
