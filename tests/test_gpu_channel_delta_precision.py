"""The chunked delta rule's (csrc/channel_delta.cu) distance from float64 beside that of the form on the fp32 pipe (recurrent_mix.cu).  At the decays that the layer has
(the reference initialisation: a rate of -1 to -16 a head, a step of 1e-3 to 0.1 a channel before the input's part) and at weaker ones it is no larger, in the
norm, for the middle token, head and key channel, and at the 99th percentile of each.  Where decays are so strong that a state holds a few tokens, both forms are two fp32 roundings (1.1e-7)
off: within a fifth in the norm, three tenths of each.  And the decays alone: a token whose key is zero leaves the state times its decays, so a state of ones holds them."""
import math

import pytest
import torch

from test_gpu_channel_delta import F64, recurrence, rel, run

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def chunked(monkeypatch):
    from nanovllm import mixops as mx
    monkeypatch.setattr(mx, "delta_pays", lambda *a: True)             # short portions too


def layer_inputs(lens, H, G, seed, shift=None):
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)
    n, D = sum(lens), 128
    step = torch.exp(torch.empty(H * D, device="cuda").uniform_(math.log(1e-3), math.log(0.1), generator=g))
    bias = step + torch.log(-torch.expm1(-step)) if shift is None else torch.full((H * D,), shift, device="cuda")
    return dict(x=torch.nn.functional.silu(r(n, (2 * G + H) * D)).bfloat16(), write=r(n, H).bfloat16(), z=r(n, H * D),
                rate=-torch.empty(H, device="cuda").uniform_(1, 16, generator=g), bias=bias, state=r(len(lens), H, D, D))


@pytest.mark.parametrize("shift", [None, -8.0, -3.0, 2.0])
@pytest.mark.parametrize("lens,H", [([16] * 16, 16), ([64] * 12, 8), ([100, 417, 33], 8), ([1500], 4)])
def test_no_further_from_float64_than_the_fp32_form(lens, H, shift):
    a = layer_inputs(lens, H, 4, sum(lens) + H, shift)
    hist = [i % 2 for i in range(len(lens))]
    want = recurrence(a, lens, hist, H, 4, 128, 128, 128 ** -0.5)
    new, old = (run(a, lens, hist, H, 4, 128, 128, 128 ** -0.5, forgetting=f) for f in (True, False))
    limit = 1.0 if shift in (None, -8.0) else 1.2
    for got, former, ref, dim in zip(new, old, want, (-1, 2)):
        assert rel(got, ref) <= limit * rel(former, ref)
        each = lambda t: ((t.to(F64) - ref).norm(dim=dim) / ref.norm(dim=dim).clamp_min(1e-30)).flatten()
        e, o = each(got), each(former)                      # of every token and head, of every key channel of every state
        assert e.median() <= (1.0 if limit == 1.0 else 1.3) * o.median() and e.quantile(0.99) <= (1.0 if limit == 1.0 else 1.3) * o.quantile(0.99)


@pytest.mark.parametrize("token", [0, 7])
def test_what_strong_decays_have_made_small_keeps_its_bits(token):
    """One token writes, the next ones' write gates are closed (a key of zeros) and every channel decays: state and read-outs are a millionth of what they were, and as
    exact.  Sixteen decays are each rounded to half a unit of 2^-24, and all the same way where all are the same: 16 x 6e-8."""
    H, D, n = 4, 128, 16
    a = layer_inputs([n], H, H, 3, 0.0)
    a["z"].fill_(0.5)
    a["rate"].fill_(-1.0)
    keep = torch.zeros(n, 1, device="cuda")
    keep[token] = 1
    a["x"][:, H * D:2 * H * D] *= keep.bfloat16()
    want = recurrence(a, [n], [0], H, H, D, D, 1.0)
    got = run(a, [n], [0], H, H, D, D, 1.0)
    assert want[1].abs().max() < 1e-3
    assert rel(got[1], want[1]) < 1.1e-6 and rel(got[0][-1], want[0][-1]) < 1.1e-6


def decays(z, rate, forgetting):
    """z [n] (a multiple of 128 x 16), one rate: the decays that the kernel forms, through one-token portions of a step."""
    D, V, H = 128, 8, 16
    tokens = z.numel() // (D * H)
    lens = [16] + [1] * tokens                              # (a longer portion takes the step to the chunked form)
    n = sum(lens)
    a = dict(x=torch.zeros(n, (2 * H * D) + H * V, device="cuda").bfloat16(), write=torch.zeros(n, H, device="cuda").bfloat16(),
             z=torch.cat((torch.zeros(16, H * D, device="cuda"), z.view(tokens, H * D))), rate=torch.full((H,), rate, device="cuda"),
             bias=torch.zeros(H * D, device="cuda"), state=torch.ones(len(lens), H, V, D, device="cuda"))
    _, state = run(a, lens, [1] * len(lens), H, H, D, V, 1.0, forgetting=forgetting)
    return state[1:, :, 0].flatten()


@pytest.mark.parametrize("rate,times", [(-1e-3, 1.01), (-0.3, 1.01), (-1.0, 1.01), (-16.0, 1.01), (-400.0, 2.0)])
def test_decays_alone(rate, times):
    """Against float64, beside the fp32 form's (expf and log1pf): no further off in the mean square (within one per cent), neither as a decay nor as what it takes
    away, 1 - g; at the ends exact.  At a rate of -400 every decay that is not zero has a softplus below 0.22, whose last bits count up to 87 times: within twice."""
    z = torch.linspace(-100, 100, 128 * 16 * 24, device="cuda")
    special = torch.tensor([0.0, -0.0, float("inf"), -float("inf"), 1e-40, -1e-40, 3e38, -3e38, 20.0, -20.0], device="cuda")
    z[-10:] = special
    z[0] = float("nan")                                   # (its head's other channels become none too: the row of the state feeds all)
    want = torch.exp(rate * torch.nn.functional.softplus(z.to(F64), threshold=1e9))
    new, old = decays(z, rate, True), decays(z, rate, False)
    assert torch.isnan(new[0]) and torch.isnan(old[0])
    z, want, new, old = (t[128:] for t in (z, want, new, old))
    fine = want > 2.0 ** -126
    assert (new[~fine] <= 2.0 ** -126).all()
    for f in (lambda t: (t - want) / want, lambda t: (t - want) / (1 - want).clamp_min(2.0 ** -24)):
        e, o = (f(t.to(F64))[fine].square().mean().sqrt() for t in (new, old))
        assert e <= times * o, (float(e), float(o))
    assert new[-7] == 1.0 and new[-8] == 0.0                # exp(rate * 0) and exp(-inf)
    assert (new <= 1.0).all()
