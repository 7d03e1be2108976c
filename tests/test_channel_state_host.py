"""Matrix-state mixers with channel decays, host side: weights are read where the layer names them."""
import torch

from nanovllm.layers.channel_state import ChannelDeltaMixer


def test_a_replaced_second_factor_is_the_one_used(monkeypatch):
    """``second`` is the layer's own dictionary: a tensor put in place of a factor counts from the next call on, in the product with an fp32 result too."""
    layer = ChannelDeltaMixer(16, dict(heads=2, kv_heads=1, dim=8, vdim=8, conv=4), 1e-6, torch.bfloat16, "cpu", ranks={"a1": 8, "g1": 8})
    monkeypatch.setattr(torch, "mm", lambda a, b, out_dtype: a.to(out_dtype) @ b.to(out_dtype))            # (the CPU has no such product)
    g = torch.Generator().manual_seed(1)
    proj = torch.randn(3, layer.in_cols, generator=g).bfloat16()
    a = layer.at["a1"][0]
    for _ in range(2):
        layer.second["a2"] = torch.randn(16, 8, generator=g).bfloat16()
        assert torch.equal(layer._second(proj, "a1", True), proj[:, a:a + 8].float() @ layer.second["a2"].float().t())
