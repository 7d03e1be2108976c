"""The convolution's history after a step: portions shorter than the taps, of a tile of tokens and one more or less, with and without inputs before them, on the
vector path (bf16), the plain one (fp32, odd channels) and the one of many taps.  The history is a copy of the inputs, so it is exact."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,channels,taps", [(torch.bfloat16, 12, 4), (torch.bfloat16, 8, 2), (torch.float32, 7, 4), (torch.bfloat16, 5, 8), (torch.float32, 6, 10),
                                                 (torch.bfloat16, 4, 1)])
def test_history_holds_the_last_inputs(dtype, channels, taps):
    from nanovllm import mixops as mx
    lens = [1, 2, 3, 31, 32, 33, 34, 63, 64, 65, 66, 70, 200]
    g = torch.Generator(device="cuda").manual_seed(taps)
    n = sum(lens)
    x = torch.randn(n, channels, device="cuda", generator=g).to(dtype)
    w = torch.randn(channels, taps, device="cuda", generator=g).to(dtype)
    hist = torch.randn(len(lens), max(taps - 1, 1), channels, device="cuda", generator=g)
    old = [i % 2 for i in range(len(lens))]                 # every other sequence goes on
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    cu, ck = [0], [0]
    for l, o in zip(lens, old):
        cu.append(cu[-1] + l)
        ck.append(ck[-1] + l + 20 * o)
    state = hist.clone()
    out = mx.causal_conv(x, w, None, state, i32(range(len(lens))), mx.StepSpans(len(lens), max(lens), i32(cu), i32(ck), None), silu=False)
    for s, l in enumerate(lens):
        before = hist[s] if old[s] else torch.zeros_like(hist[s])
        seen = torch.cat((before[:taps - 1], x[cu[s]:cu[s + 1]].float()))
        if taps > 1:
            assert torch.equal(state[s], seen[-(taps - 1):])
        want = (seen.double().unfold(0, taps, 1) * w.double()).sum(-1)
        assert (out[cu[s]:cu[s + 1]].double() - want).norm() <= (1e-6 if dtype == torch.float32 else 4e-3) * want.norm()      # fp32 sums; bf16 results
