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


def grouped_choice(key, groups, keep, top):
    """The experts in the order of choice: the largest keys (NaN: minus infinity) within the ``keep`` groups whose largest keys are the largest, the lowest index among equals."""
    E = len(key)
    key = [-math.inf if v != v else v for v in key]
    size = E // groups
    tops, shut = [max(key[i * size:(i + 1) * size]) for i in range(groups)], [groups > 1 and keep < groups] * groups
    waiting = [True] * groups
    for _ in range(keep if keep < groups else 0):
        i, _ = best(tops, waiting)
        waiting[i] = shut[i] = False
    open_, chosen = [not shut[e // size] for e in range(E)], []
    for _ in range(top):
        e, _ = best(key, open_)
        open_[e] = False
        chosen.append(e)
    return chosen


def grouped_case(E, sigmoid):
    """Logits and corrections whose keys are equal to the last bit or 5e-6 apart, in float64 and in the kernel's fp32 alike: whole numbers and a few special ones; their sigmoids are
    0, 1/2, 1 or irrational, the corrections quarters (0 beside softmax scores).  A NaN or +inf among a row's logits leaves no softmax score."""
    g = torch.Generator().manual_seed(E + sigmoid)
    z = torch.randint(-3, 4, (29, E), generator=g).double()
    special = torch.tensor([0.0, -0.0, 1e-40, math.inf, -math.inf, math.nan, 3.4e38] if sigmoid else [0.0, -0.0, -math.inf]).double()
    pick = special[torch.randint(0, len(special), (29, E), generator=g)]
    z = torch.where(torch.rand(29, E, generator=g) < 0.2, pick, z)
    z[0] = 1.0                                                              # nothing but equals
    z[1] = -math.inf if sigmoid else 2.0
    z[2, E // 2] = math.nan
    z[3, E - 1] = math.inf if sigmoid else z[3, E - 1]
    corr = torch.randint(-2, 3, (E,), generator=g).double() / 4 if sigmoid else torch.zeros(E).double()
    corr[0] = -0.0
    score = torch.sigmoid(z) if sigmoid else torch.softmax(z, -1)
    return z.float(), corr.float(), score, score + corr


CASES = [(40, 8, 4, 4, 32), (20, 4, 2, 2, 16), (33, 1, 1, 4, 33), (96, 3, 2, 8, 90), (1024, 64, 5, 6, 1000), (12, 4, 1, 3, 12), (40, 8, 2, 6, 32), (20, 4, 1, 4, 16)]


@pytest.mark.parametrize("sigmoid", [False, True])
@pytest.mark.parametrize("renorm", [False, True])
@pytest.mark.parametrize("E,groups,keep,top,real", CASES)
def test_best_groups_then_largest_scores(E, groups, keep, top, real, renorm, sigmoid):
    from nanovllm import mixops as mx
    z, corr, score, key = grouped_case(E, sigmoid)
    idx, w = mx.moe_route_grouped(z.cuda(), E, top, corr.cuda(), groups, keep, real, sigmoid=sigmoid, renorm=renorm, scale=1.5)
    otherwise = 0
    for t in range(z.shape[0]):
        apart = key[t].unique()
        assert not (apart.diff() < 5e-6).any()                              # no choice hangs on rounding (2^-23 of 1 at most)
        chosen = grouped_choice(key[t].tolist(), groups, keep, top)
        otherwise += chosen != grouped_choice(key[t].tolist(), 1, 1, top)
        assert idx[t].tolist() == [e if e < real else -1 for e in chosen], t
        want = score[t, chosen] * 1.5 / (score[t, chosen].sum() + 1e-20 if renorm else 1.0)
        assert torch.allclose(w[t].cpu().double(), want, rtol=1e-5, atol=1e-30, equal_nan=True), t
    assert otherwise or keep >= top or groups == 1 or E > 1000              # closed groups hold what would be chosen without them
