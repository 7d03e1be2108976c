"""Row-wise kernels with wide accesses: widths around what a lane holds, rows that do not fill a CTA, and strides or starts that keep the element-wise form.

Reference: float64 on the same values; one bf16 step where a rounding falls on the other side."""
import pytest
import torch

from test_gpu_kernels import assert_close_bf16, bf

pytestmark = pytest.mark.gpu
EPS = 1e-6


@pytest.fixture(scope="module")
def mx():
    from nanovllm import mixops
    return mixops


@pytest.mark.parametrize("rows,cols", [(1, 8), (5, 256), (3, 264), (7, 512), (130, 520), (2, 1024), (9, 1032), (4, 2048), (4, 2056), (3, 100)])
@pytest.mark.parametrize("pad,off", [(0, 0), (8, 8), (4, 0), (0, 1)])
def test_rmsnorm(mx, rows, cols, pad, off):
    x, w = bf(rows, cols + pad + off, seed=1), 1 + 0.1 * bf(cols, seed=2)
    view = x.cuda()[:, off:]
    want = x[:, off:off + cols].double()
    want = want / (want.square().mean(-1, keepdim=True) + EPS).sqrt() * w.double()
    assert_close_bf16(mx.rmsnorm(view, w.cuda(), EPS, cols=cols), want.to(torch.bfloat16), "rmsnorm", ulps=1.01)


@pytest.mark.parametrize("rank,rd,rot", [(512, 64, 64), (256, 64, 64), (8, 16, 8), (256, 64, 32), (512, 60, 60), (520, 64, 64)])
@pytest.mark.parametrize("layout", [0, 1])
def test_latent_store(mx, rank, rd, rot, layout):
    from nanovllm.layers.rotary_embedding import build_banded_cos_sin
    n = 13
    dkv, w = bf(n, rank + rd + 24, seed=3), 1 + 0.1 * bf(rank, seed=4)
    cs = build_banded_cos_sin(rot, 256, 1e4, None, "cuda")
    pos = torch.arange(n) * 9
    slots = torch.randperm(40, generator=torch.Generator().manual_seed(5))[:n].to(torch.int32)
    slots[4] = -1
    cache = torch.full((40, rank + rd), 7.0, dtype=torch.bfloat16, device="cuda")
    mx.latent_store(dkv.cuda(), w.cuda(), cs, pos.cuda(), slots.cuda(), cache, rank, rd, EPS, layout)
    lat = dkv[:, :rank].double()
    want = torch.full((40, rank + rd), 7.0, dtype=torch.float64)
    r = dkv[:, rank:rank + rd].double()
    c, s = cs.cpu()[pos, :rot // 2].double(), cs.cpu()[pos, rot // 2:].double()
    lo, hi = (slice(0, rot, 2), slice(1, rot, 2)) if layout == 0 else (slice(0, rot // 2), slice(rot // 2, rot))
    u, v = r[:, lo].clone(), r[:, hi].clone()
    r[:, lo], r[:, hi] = u * c - v * s, v * c + u * s
    row = torch.cat((lat / (lat.square().mean(-1, keepdim=True) + EPS).sqrt() * w.double(), r), -1)
    ok = slots >= 0
    want[slots[ok].long()] = row[ok]
    assert_close_bf16(cache, want.to(torch.bfloat16), "latent store", ulps=1.01)


@pytest.mark.parametrize("n,H,vdim", [(1, 3, 128), (37, 5, 68), (700, 16, 128), (601, 16, 100), (9, 2, 64), (9, 2, 66), (3, 2, 132)])
@pytest.mark.parametrize("shared,silu,gated", [(True, True, True), (False, False, True), (True, True, False)])
def test_head_norm_gate(mx, n, H, vdim, shared, silu, gated):
    x, w, gate = bf(n, H, vdim, seed=6).float(), 1 + 0.1 * bf(vdim if shared else H * vdim, seed=7), bf(n, H * vdim + 8, seed=8)
    got = mx.head_rmsnorm_gate(x.cuda(), w.cuda(), gate.cuda()[:, :H * vdim] if gated else None, EPS, torch.bfloat16, silu=silu, out_scale=0.5)
    z = gate[:, :H * vdim].double()
    want = x.double() / (x.double().square().mean(-1, keepdim=True) + EPS).sqrt() * 0.5 * (w.double() if shared else w.double().view(H, vdim))
    want = want.view(n, -1) * ((torch.nn.functional.silu(z) if silu else z.sigmoid()) if gated else 1)
    assert_close_bf16(got, want.to(torch.bfloat16), "head norm gate", ulps=1.01)
