"""Single tokens over windows: pages whose rows a warp addresses in one go (multiples of sixteen, powers of two) and pages looked up row by row have the
same result, bit for bit, and both are as near to float64 as the other forms of this layer (csrc/window_attn.cu, the key-sharing form)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
LENS = [0, 1, 15, 16, 17, 63, 64, 65, 80, 128, 129, 191, 200, 333]          # edges of a warp's sixteen keys and of the tiles of 64, a padding row


def exact(q, k, v, scale, slopes, window, keep):
    """One query over float64 rows [keys, d], per head of its group."""
    j, pos = torch.arange(k.shape[0]), k.shape[0] - 1
    s = q @ k.t() * scale - slopes[:, None] * (pos - j)
    if window:
        s = s.masked_fill((pos - j >= window) & (j >= keep), -torch.inf)
    return torch.softmax(s, 1) @ v


@pytest.mark.parametrize("splits", [1, 3])
@pytest.mark.parametrize("shape", [(16, 8, 128, 128, 0, 0), (16, 8, 128, 128, 100, 0), (8, 1, 64, 128, 70, 20), (16, 1, 32, 32, 0, 0), (6, 2, 96, 40, 64, 0), (4, 4, 64, 64, 130, 5)])
def test_pages_of_any_size(shape, splits):
    from nanovllm import mixops
    H, G, d, vd, window, keep = shape
    g = torch.Generator().manual_seed(H * 1000 + d + window)
    rows = [torch.randn(n, G * (d + vd), generator=g).bfloat16() for n in LENS]
    q, slopes = torch.randn(len(LENS), H * d, generator=g).bfloat16(), torch.rand(H, generator=g) * 0.1
    spans = mixops.StepSpans(len(LENS), 1, None, None, torch.tensor(LENS, dtype=torch.int32).cuda())
    results = []
    for bs in (16, 64, 8, 48):                              # in one go, in one go, row by row by shifts, row by row by division
        width = -(-max(LENS) // bs)
        tables = torch.randperm(len(LENS) * width, generator=g).view(len(LENS), width)
        cache = torch.full((len(LENS) * width * bs, G * (d + vd)), float("nan"), dtype=torch.bfloat16)       # no row past an end may count
        for s, r in enumerate(rows):
            at = torch.arange(r.shape[0])
            cache[tables[s][at // bs] * bs + at % bs] = r
        results.append(mixops.window_attention(q.cuda(), cache.cuda(), tables.int().cuda(), bs, spans, H, G, d, vd, d ** -0.5, slopes.cuda(), window,
                                               keep_first=keep, splits=splits, out_f32=True).cpu())
    live = [s for s, n in enumerate(LENS) if n]
    for other in results[1:]:
        assert torch.equal(results[0][live], other[live])
    got, want = results[0].double().view(len(LENS), H, vd), torch.zeros(len(LENS), H, vd, dtype=torch.float64)
    rep = H // G
    for s in live:
        k, v = rows[s][:, :G * d].double(), rows[s][:, G * d:].double()
        for h in range(G):
            here = slice(h * rep, (h + 1) * rep)
            want[s, here] = exact(q[s].view(H, d)[here].double(), k[:, h * d:(h + 1) * d], v[:, h * vd:(h + 1) * vd], d ** -0.5, slopes[here].double(), window, keep)
    # weights are rounded to bf16, each by 2^-9 of itself at most: so is what they leave of a result, against the sum of the magnitudes
    size = torch.stack([torch.stack([rows[s][:, G * d:].double().abs().max() for _ in range(H)]) for s in live])[:, :, None]
    assert ((got[live] - want[live]).abs() <= 2.0 ** -8 * size).all()
