"""Chunked form of the delta rule with channel decays (csrc/channel_delta.cu) against the recurrence in float64: lengths around a chunk and around the
launch pairs' boundaries, sizes that leave tiles partly empty, decays from none to all, states in memory; tokens that are no numbers.

The tolerance: operands carry 22 to 23 bits, so a product of 128 terms is off by some 2^-22; over a sequence such errors add up like a random walk
while the state forgets.  2e-6 of the result's norm is eight of them (measured: 1e-7 to 8e-7, the fp32-pipe form 1e-7 to 3e-6)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
F64 = torch.float64


def inputs(lens, H, G, D, V, seed, shift):
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)
    n = sum(lens)
    return dict(x=r(n, 2 * G * D + H * V).bfloat16(), write=(2 * r(n, H)).bfloat16(), z=r(n, H * D) + shift, rate=-torch.linspace(0.3, 8.0, H, device="cuda"),
                bias=0.5 * r(H * D), state=r(len(lens), H, V, D))


def recurrence(a, lens, hist, H, G, D, V, scale):
    x = a["x"].to(F64)
    per = lambda t: t.view(-1, G, D).repeat_interleave(H // G, 1)
    q, k, v = per(x[:, :G * D]), per(x[:, G * D:2 * G * D]), x[:, 2 * G * D:].reshape(-1, H, V)
    q, k = (t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6) for t in (q, k))
    beta = torch.sigmoid(a["write"].to(F64))
    decay = torch.exp(a["rate"].to(F64)[:, None] * torch.nn.functional.softplus((a["z"].to(F64) + a["bias"].to(F64)).view(-1, H, D)))
    out, state, at = torch.empty_like(v), a["state"].to(F64).clone(), 0
    for s, n in enumerate(lens):
        S = state[s] if hist[s] else torch.zeros_like(state[s])
        for t in range(at, at + n):
            S = S * decay[t][:, None]
            S = S + (beta[t][:, None] * (v[t] - (S @ k[t][..., None])[..., 0]))[..., None] * k[t][:, None]
            out[t] = (S @ q[t][..., None])[..., 0] * scale
        state[s], at = S, at + n
    return out, state


def run(a, lens, hist, H, G, D, V, scale, forgetting=True):
    from nanovllm import mixops as mx
    n = len(lens)
    cu, ck = [0], [0]
    for i, l in enumerate(lens):
        cu.append(cu[-1] + l)
        ck.append(ck[-1] + l + (9 if hist[i] else 0))
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    slots = list(range(n))[::-1]
    state = a["state"].flip(0).contiguous()
    out = mx.channel_state(a["x"], 0, G * D, 2 * G * D, a["write"], a["z"].clone(), a["rate"], a["bias"], 1.0, state, i32(slots),
                           mx.StepSpans(n, max(lens), i32(cu), i32(ck), None), H, G, D, V, scale, forgetting=forgetting)
    return out, state.flip(0)


rel = lambda a, b: ((a.to(F64) - b).norm() / b.norm()).item()


@pytest.mark.parametrize("shift", [-8.0, -3.0, 2.0])
@pytest.mark.parametrize("lens,hist,H,G,D,V", [
    ([1, 15, 16, 17, 129], [0, 1, 1, 0, 1], 4, 2, 128, 128),
    ([31, 200], [1, 0], 3, 3, 72, 40),
    ([160], [1], 2, 1, 120, 8),
    ([140, 2, 33], [0, 0, 1], 2, 2, 128, 200)])
def test_against_the_recurrence(lens, hist, H, G, D, V, shift):
    from nanovllm import mixops as mx
    assert mx.delta_chunks(max(lens), D)
    a = inputs(lens, H, G, D, V, sum(lens) + H, shift)
    want = recurrence(a, lens, hist, H, G, D, V, D ** -0.5)
    got = run(a, lens, hist, H, G, D, V, D ** -0.5)
    assert rel(got[0], want[0]) < 2e-6 and rel(got[1], want[1]) < 2e-6


def test_several_launch_pairs(monkeypatch):
    """A step whose chunks do not fit the workspace's bound is cut, the state going through memory in between."""
    from nanovllm import _native as nat, mixops as mx
    H, G, D, V, lens = 64, 64, 128, 16, [700] * 6
    row = nat.load_mix().b200m_channel_delta_workspace_bytes(0, 1, H)
    monkeypatch.setattr(mx, "DELTA_WORKSPACE", 100 * row)   # 262 + 6 rows
    a = inputs(lens, H, G, D, V, 5, -4.0)
    got, state = run(a, lens, [0] * 6, H, G, D, V, 1.0)
    want, wstate = run(a, lens, [0] * 6, H, G, D, V, 1.0, forgetting=False)
    assert rel(got, want.to(F64)) < 4e-6 and rel(state, wstate.to(F64)) < 4e-6        # two forms, each within 2e-6


@pytest.mark.parametrize("part", ["q", "k", "v", "z", "write"])
def test_what_is_no_number_reaches_no_earlier_token(part):
    H, G, D, V, n = 2, 1, 128, 128, 150
    a = inputs([n], H, G, D, V, 3, -3.0)
    want, _ = run(a, [n], [1], H, G, D, V, 1.0)
    bad = 37                                                # inside a chunk
    if part == "z":
        a["z"][bad, 5] = float("nan")
    elif part == "write":
        a["write"][bad, 0] = float("nan")
    else:
        a["x"][bad, {"q": 3, "k": G * D + 3, "v": 2 * G * D + 3}[part]] = float("inf" if part == "v" else "nan")
    got, state = run(a, [n], [1], H, G, D, V, 1.0)
    assert (got[:bad] - want[:bad]).norm() <= 1e-6 * want[:bad].norm()
    if part == "q":                                         # a query alone: its own token, nothing after
        assert not torch.isfinite(got[bad]).any() and torch.isfinite(state).all()
        assert (got[bad + 1:] - want[bad + 1:]).norm() <= 1e-6 * want[bad + 1:].norm()
    else:
        assert not torch.isfinite(got[bad + 1:, 0]).all() and not torch.isfinite(state[0, 0]).all()
    if part == "v":                                         # a value's column alone
        cols = [c for c in range(V) if c != 3]
        assert torch.isfinite(got[:, :, cols]).all()
