"""Packed prompts whose K and V are scattered inside the attention launch (csrc/fa_tc.cuh): results and cache are those of the two launches, bit for bit; one
token, odd row counts, shares of no row, of one and of many, head groups of 1 to 4, slots that are not stored, projections side by side and apart."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lens", [[1], [2, 1], [17, 33, 64], [128] * 5, [300, 1, 511], [1500, 700], [64] * 200])
@pytest.mark.parametrize("hq,hkv", [(8, 8), (16, 8), (6, 2), (4, 1), (3, 1)])
@pytest.mark.parametrize("apart,block", [(False, 16), (True, 256)])
def test_same_as_two_launches(lens, hq, hkv, apart, block, monkeypatch):
    from nanovllm import ops
    D, n = 128, sum(lens)
    g = torch.Generator(device="cuda").manual_seed(n + hq)
    kv = torch.zeros(ops.kv_cache_shape(2, -(-n // block) + 3, hkv, block, D), dtype=torch.bfloat16, device="cuda")
    ops.bind_kv_cache(kv)
    qkv = torch.randn(n, (hq + 2 * hkv) * D, device="cuda", generator=g).bfloat16()
    q, k, v = (t.view(n, -1, D) for t in qkv.split((hq * D, hkv * D, hkv * D), 1))
    if apart:
        k, v = k.contiguous(), v.contiguous()
    slots = torch.randperm(kv.shape[2] * block, device="cuda", generator=g)[:n].to(torch.int32)
    slots[::7] = -1
    cu = torch.tensor([0] + lens).cumsum(0).to(torch.int32).cuda()
    got = []
    for inside in (True, False):
        kv.zero_()
        monkeypatch.setattr(ops, "prefill_hides_store", lambda *a: inside)
        before = ops.LAUNCHES[0]
        out = ops.paged_prefill_store(1, q, k, v, slots, cu, cu, max(lens), max(lens), D ** -0.5)
        assert ops.LAUNCHES[0] - before == (1 if inside else 2)
        got.append((out, kv.clone()))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
    assert got[0][1][:, 1].any() or n == 1
