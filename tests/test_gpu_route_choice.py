"""The routers' choice (csrc/moe.cu) against a plain loop: equal logits, zeros of either sign, subnormal numbers, infinities and NaN, more experts than lanes, closed groups."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def logits(n, E, seed):
    g = torch.Generator().manual_seed(seed)
    z = torch.randint(-3, 4, (n, E), generator=g).float()                   # many equal ones
    special = torch.tensor([0.0, -0.0, 1e-40, -1e-40, math.inf, -math.inf, math.nan, 3.4e38])
    pick = torch.randint(0, len(special), (n, E), generator=g)
    return torch.where(torch.rand(n, E, generator=g) < 0.3, special[pick], z)


def best(values, open_):
    """The largest open value (NaN: minus infinity), among equals the first."""
    at, top = -1, -math.inf
    for e, v in enumerate(values):
        v = -math.inf if v != v else v
        if open_[e] and (at < 0 or v > top):
            at, top = e, v
    return at, top


@pytest.mark.parametrize("E,top", [(1, 1), (16, 2), (33, 4), (64, 8), (1000, 3)])
def test_largest_logits(E, top):
    from nanovllm import mixops as mx
    z = logits(37, E, E)
    idx, w = mx.moe_route(z.cuda(), E, top)
    for t in range(z.shape[0]):
        open_ = [True] * E
        for k in range(top):
            e, v = best(z[t].tolist(), open_)
            open_[e] = False
            assert idx[t, k].item() == e
            assert w[t, k].item() == pytest.approx(1 / (1 + math.exp(-v)) if v > -80 else 0.0, rel=1e-5, abs=1e-30)


@pytest.mark.parametrize("E,groups,keep,top,real", [(40, 8, 4, 4, 32), (20, 4, 2, 2, 16), (33, 1, 1, 4, 33), (96, 3, 2, 8, 90), (1024, 64, 5, 6, 1000)])
def test_best_groups_then_largest_scores(E, groups, keep, top, real):
    from nanovllm import mixops as mx
    g = torch.Generator().manual_seed(E)
    z = torch.randint(-4, 5, (29, E), generator=g).float()
    corr = torch.randint(-2, 3, (E,), generator=g).float() / 4
    corr[0] = -0.0
    idx, w = mx.moe_route_grouped(z.cuda(), E, top, corr.cuda(), groups, keep, real, scale=1.5)
    p = torch.softmax(z.cuda(), -1).cpu()                                   # scores far enough apart, or equal to the last bit: the choice does not hang on rounding
    size = E // groups
    for t in range(z.shape[0]):
        key = [(round(a, 5)) for a in (p[t] + corr).tolist()]
        tops = [max(key[i * size:(i + 1) * size]) for i in range(groups)]
        open_groups, shut = [True] * groups, [True] * groups
        for _ in range(keep):
            i, _ = best(tops, open_groups)
            open_groups[i], shut[i] = False, False
        open_ = [groups == 1 or keep >= groups or not shut[e // size] for e in range(E)]
        chosen = []
        for _ in range(top):
            e, _ = best(key, open_)
            open_[e] = False
            chosen.append(e)
        got = idx[t].tolist()
        ties = len({round(key[e], 4) for e in range(E)}) < E
        want_keys = [key[e] for e in chosen]
        assert [i for i in got] == [e if e < real else -1 for e in chosen] or (ties and sorted(key[e] for e in got if e >= 0) == sorted(k for e, k in zip(chosen, want_keys) if e < real))
        total = sum(p[t, e].item() for e in chosen)
        for k, e in enumerate(chosen):
            if got[k] == e:
                assert w[t, k].item() == pytest.approx(1.5 * p[t, e].item() / total, rel=1e-4)
