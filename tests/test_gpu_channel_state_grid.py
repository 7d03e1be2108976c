"""Delta rule over prompt portions on both sides of the rule that gives a CTA all of an SM's registers: a step of many sequences against the same sequences
in steps of two.  The arithmetic and its order are the same, so the results agree to fp32 rounding (contraction of products may differ between instances)."""
import pytest
import torch

from test_gpu_kernels import bf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,G,vdim", [(16, 4, 64), (8, 8, 100)])
def test_many_sequences_as_few(H, G, vdim):
    from nanovllm import mixops as mx
    D, lens = 128, [5 + 3 * i for i in range(20)]
    assert H * len(lens) * -(-vdim // 64) > 148 >= H * 2 * -(-vdim // 64)
    n, qk = sum(lens), G * D
    x, write, dec = bf(n, 2 * qk + H * vdim, seed=1).cuda(), bf(n, H, seed=2).cuda(), bf(n, H * D, seed=3).float().cuda()
    rate, bias = -torch.linspace(0.5, 2, H).cuda(), bf(H * D, seed=4).float().cuda()
    start = bf(len(lens), H, vdim, D, seed=5).float().cuda() * 0.1

    def run(seqs):
        first = sum(lens[:seqs[0]])
        part = [lens[i] for i in seqs]
        rows = slice(first, first + sum(part))
        cu = torch.tensor([0] + part).cumsum(0).to(torch.int32)
        ck = torch.tensor([0] + [l + 7 for l in part]).cumsum(0).to(torch.int32)             # seven tokens before: the state in memory counts
        spans = mx.StepSpans(len(part), max(part), cu.cuda(), ck.cuda(), None)
        state, slots = start[seqs[0]:seqs[-1] + 1].clone(), torch.arange(len(part), dtype=torch.int32).cuda()
        out = mx.channel_state(x[rows], 0, qk, 2 * qk, write[rows], dec[rows].clone(), rate, bias, 1.0, state, slots, spans, H, G, D, vdim, D ** -0.5)
        return out, state

    out, state = run(list(range(len(lens))))
    few = [run([i, i + 1]) for i in range(0, len(lens), 2)]
    for got, want in ((out, torch.cat([f[0] for f in few])), (state, torch.cat([f[1] for f in few]))):
        assert torch.isfinite(got).all()
        assert (got - want).abs().max().item() <= 1e-5 * want.abs().max().item()
