"""Which CTA takes which item of a prompt step (csrc/fa_tc.cuh deals them out round by round, every other round from the far end): numbers of items around whole rounds, each item
done once.  Reference: the same attention in float64 (P is rounded to bf16, 2^-9 relative, and so is the result)."""
import pytest
import torch

from test_gpu_kernels import assert_close_bf16, bf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rounds", [0, 1, 2, 3])
@pytest.mark.parametrize("more", [-1, 0, 1, 70])
def test_every_item_once(rounds, more):
    from nanovllm import ops
    from nanovllm import _native as nat
    n, l, hq = rounds * nat.handle().sm_count + more, 3, 2                # one item a sequence: two heads of one kv head
    if n <= 0:
        n = 1
    kv = torch.zeros(ops.kv_cache_shape(1, 1, 1, 16, 128), dtype=torch.bfloat16, device="cuda")
    ops.bind_kv_cache(kv)
    q, k, v = bf(n * l, hq, 128, seed=1).cuda(), bf(n * l, 1, 128, seed=2).cuda(), bf(n * l, 1, 128, seed=3).cuda()
    cu = torch.arange(0, (n + 1) * l, l, dtype=torch.int32, device="cuda")
    got = ops.paged_prefill(0, q, k, v, cu, cu, l, l, 128 ** -0.5, out=torch.full_like(q, float("nan")))
    s = torch.einsum("nihd,njd->nhij", q.view(n, l, hq, 128).double(), k.view(n, l, 128).double()) * 128 ** -0.5
    s.masked_fill_(torch.ones(l, l, dtype=torch.bool, device="cuda").triu(1), float("-inf"))
    want = torch.einsum("nhij,njd->nihd", torch.softmax(s, -1), v.view(n, l, 128).double()).reshape(n * l, hq, 128)
    assert_close_bf16(got, want.float(), f"{n} items", rel_l2=6e-3, ulps=3.0)
