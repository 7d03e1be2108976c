"""Queries and keys normalised over the whole projection, keys and values to their cache rows (bf16): columns around what the threads of a block hold in
registers, against float64.  A bf16 result has 8 significant bits, its rounding is at most half a unit of the last, 2^-8 of the element (at 1 + 2^-8); fp32 sums of at
most 4104 squares add 8e-6.  Values are copied."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("qc,kc,vc", [(8, 8, 8), (2048, 1024, 1024), (2040, 1032, 1016), (2056, 8, 16), (4096, 2048, 8), (4096, 3072, 1024), (4104, 8, 8), (64, 4096, 8), (640, 0, 0), (128, 0, 256)])
@pytest.mark.parametrize("norm_q,norm_k", [(True, True), (False, True), (True, False)])
def test_against_float64(qc, kc, vc, norm_q, norm_k):
    from nanovllm import mixops
    g = torch.Generator(device="cuda").manual_seed(qc + kc)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)
    n, cols = 11, qc + kc + vc
    x = (r(n, cols + 8) * torch.linspace(0.2, 4, cols + 8, device="cuda")).bfloat16()[:, :cols]
    wq, wk = (1 + 0.3 * r(qc)).bfloat16(), (1 + 0.3 * r(kc)).bfloat16()
    slots = torch.tensor([4, 0, 17, -1, 3, 9, 8, 30, 1, -1, 31], dtype=torch.int32, device="cuda")
    cache = torch.full((32, kc + vc), 7.0, dtype=torch.bfloat16, device="cuda") if kc + vc else None
    want, old = x.double(), x.clone()
    unit = lambda t, w: t / (t.square().mean(-1, keepdim=True) + 1e-5).sqrt() * w.double()
    mixops.qk_norm_store(x, qc, kc, vc, wq if norm_q else None, wk if norm_k and kc else None, slots if kc + vc else None, cache, 1e-5)
    close = lambda got, ref: bool(((got.double() - ref).abs() <= (2 ** -8 + 8e-6) * ref.abs()).all())
    assert close(x[:, :qc], unit(want[:, :qc], wq)) if norm_q else torch.equal(x[:, :qc], old[:, :qc])
    assert torch.equal(x[:, qc:], old[:, qc:])
    for t, s in enumerate(slots.tolist() if kc + vc else []):
        if s < 0:
            continue
        k = want[t, qc:qc + kc]
        assert close(cache[s, :kc], unit(k, wk)) if norm_k and kc else torch.equal(cache[s, :kc], old[t, qc:qc + kc])
        assert torch.equal(cache[s, kc:], old[t, qc + kc:])
    if kc + vc:
        rest = [s for s in range(32) if s not in slots.tolist()]
        assert bool((cache[rest] == 7.0).all())
