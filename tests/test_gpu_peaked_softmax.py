"""Rows whose softmax is peaked: the weights of the largest keys carry the result, so a softmax reference that lags behind a row's maximum shows as
rounding of those weights (csrc/fa_tc.cuh, FaParams::lag; csrc/latent_decode.cu).

Bound: the error against float64 of the same steps in torch, with the weights formed against the exact maximum and rounded to bf16 as the mma.sync
forms of these layers do, and a tenth more for sums in another order.  A lag of 2^8 is 1.4 to 2.8 times that error at these deviations."""
import pytest
import torch

from test_gpu_kernels import bf, make_tables

pytestmark = pytest.mark.gpu
LOG2E = 1.4426950408889634


def rounded(x):
    return x.to(torch.bfloat16).double()


def running(scores, values, block=64):
    """float64 scores (natural units, -inf where hidden) of one head [rows, keys]: what bf16 weights against the running maximum give."""
    m, l = torch.full_like(scores[:, :1], -torch.inf), torch.zeros_like(scores[:, :1])
    o = torch.zeros(scores.shape[0], values.shape[1], dtype=torch.float64, device=scores.device)
    for a in range(0, scores.shape[1], block):
        s = scores[:, a:a + block]
        new = torch.maximum(m, s.max(1, keepdim=True).values)
        f = torch.where(new == m, torch.ones_like(m), torch.exp(m - new))
        p = torch.where(s == -torch.inf, torch.zeros_like(s), torch.exp(s - torch.where(new == -torch.inf, torch.zeros_like(new), new)))
        l, o, m = l * f + p.sum(1, keepdim=True), o * f + rounded(p) @ values[a:a + block], new
    return o / l


def causal(scores, off, window):
    i, j = off + torch.arange(scores.shape[0], device=scores.device)[:, None], torch.arange(scores.shape[1], device=scores.device)[None, :]
    return scores.masked_fill((j > i) | (i - j >= (window or 1 << 30)), -torch.inf)


def relative(a, b):
    return ((a.double() - b).norm() / b.norm()).item()


def cu(lens):
    return torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32).cuda()


def paged(rows, lens, bs, seed):
    nblk = sum(-(-c // bs) for c in lens)
    tables = make_tables(lens, bs, nblk, seed=seed)
    cache = torch.zeros(nblk * bs, rows.shape[1], dtype=torch.bfloat16, device="cuda")
    at = 0
    for i, c in enumerate(lens):
        p = torch.arange(c)
        cache[(tables[i][p // bs].long() * bs + p % bs).cuda()] = rows[at:at + c]
        at += c
    return cache, tables.cuda()


@pytest.mark.parametrize("deviation", [1.0, 2.0, 5.0])
@pytest.mark.parametrize("window", [0, 700])
@pytest.mark.parametrize("slopes", [False, True])
def test_windowed_prompts(deviation, window, slopes):
    from nanovllm import mixops as mx
    H, G, scale, lens, new = 4, 2, deviation / 128 ** 0.5, [1500, 900], [1500, 300]
    q, rows = bf(sum(new), H * 128, seed=1).cuda(), bf(sum(lens), G * 256, seed=2).cuda()
    cache, tables = paged(rows, lens, 64, 3)
    bias = torch.linspace(0.001, 0.004, H).cuda() if slopes else None
    spans = mx.StepSpans(2, max(new), cu(new), cu(lens), None)
    got = mx.window_attention(q, cache, tables, 64, spans, H, G, 128, 128, scale, slopes=bias, window=window, out_f32=True)
    want, sim, qa, ka = [], [], 0, 0
    for n, l in zip(new, lens):
        for h in range(H):
            k, v = rows[ka:ka + l, h // 2 * 128:][:, :128].double(), rows[ka:ka + l, G * 128 + h // 2 * 128:][:, :128].double()
            s = q[qa:qa + n, h * 128:][:, :128].double() @ k.T * scale
            if slopes:
                s = s - bias[h].double() * ((l - n + torch.arange(n, device="cuda"))[:, None] - torch.arange(l, device="cuda")[None, :])
            s = causal(s, l - n, window)
            want.append(torch.softmax(s, -1) @ v)
            sim.append(running(s, v))
        qa, ka = qa + n, ka + l
    cut = lambda parts: torch.cat([torch.cat(parts[:H], 1), torch.cat(parts[H:], 1)])
    want, sim = cut(want), cut(sim)
    assert relative(got, want) <= 1.1 * relative(sim, want), (relative(got, want), relative(sim, want))


@pytest.mark.parametrize("deviation", [2.0, 5.0])
def test_latent_prompts(deviation):
    """Keys, values and the result are bf16 on both sides; the rotation is the identity (position 0 of the table for every token)."""
    from nanovllm import mixops as mx
    H, d, rd, R, lens = 2, 128, 64, 256, [1400, 333]
    n, scale = sum(lens), deviation / 192 ** 0.5
    q, rows = bf(n, H, d + rd, seed=4).cuda(), bf(n, R + rd, seed=5).cuda()
    w = bf(H * (d + 128), R, scale=R ** -0.5, seed=6).cuda()
    cache, tables = paged(rows, lens, 256, 7)
    cs = torch.cat((torch.ones(1, rd // 2), torch.zeros(1, rd // 2)), 1).cuda()
    spans, pos = mx.StepSpans(2, max(lens), cu(lens), cu(lens), None), torch.zeros(n, dtype=torch.int64).cuda()
    kv = torch.nn.functional.linear(rows[:, :R], w)
    got = mx.latent_prompt(q.clone(), w, d, 128, cache, tables, 256, spans, None, cs, pos, scale)
    want, sim, at = [], [], 0
    for l in lens:
        for h in range(H):
            k = torch.cat((kv[at:at + l, h * d:][:, :d], rows[at:at + l, R:]), 1).double()
            v = kv[at:at + l, H * d + h * 128:][:, :128].double()
            s = causal(q[at:at + l, h].double() @ k.T * scale, 0, 0)
            want.append(torch.softmax(s, -1) @ v)
            sim.append(rounded(running(s, v)))
        at += l
    cut = lambda parts: torch.cat([torch.cat(parts[:H], 1), torch.cat(parts[H:], 1)])
    want, sim = cut(want), cut(sim)
    assert relative(got, want) <= 1.1 * relative(sim, want), (relative(got, want), relative(sim, want))


@pytest.mark.parametrize("deviation", [1.0, 5.0])
@pytest.mark.parametrize("lens", [[3000, 700, 129], [8000]])
def test_latent_decode(deviation, lens):
    """Two bf16 terms hold the weights here: what is left is the rounding of the result."""
    from nanovllm import mixops as mx
    H, rd, R, n = 16, 64, 512, len(lens)
    rows, scale = bf(sum(lens), R + rd, seed=8).cuda(), deviation / (R + rd) ** 0.5
    cache, tables = paged(rows, lens, 128, 9)
    q_lat, q_raw = bf(H, n, R, seed=10).cuda(), bf(n, H, rd, seed=11).cuda()
    cs = torch.cat((torch.ones(1, rd // 2), torch.zeros(1, rd // 2)), 1).expand(max(lens), -1).contiguous().cuda()
    spans = mx.StepSpans(n, 1, None, None, torch.tensor(lens, dtype=torch.int32).cuda())
    got = mx.latent_attention(q_lat, q_raw, 0, cache, tables, 128, spans, None, cs, scale)
    want, at = torch.empty(H, n, R, dtype=torch.float64, device="cuda"), 0
    for i, l in enumerate(lens):
        c = rows[at:at + l].double()
        want[:, i] = torch.softmax(torch.cat((q_lat[:, i], q_raw[i]), -1).double() @ c.T * scale, -1) @ c[:, :R]
        at += l
    assert relative(got, want) <= 1.1 * relative(rounded(want), want), (relative(got, want), relative(rounded(want), want))
