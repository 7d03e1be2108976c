"""Matrix-state mixers with channel decays, host side: weights are read where the layer names them; which prompt steps run in chunks, and what those hold."""
import pytest
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


@pytest.mark.parametrize("lens,heads,chunked", [
    ([2048] * 4, 16, True), ([4096], 8, True), ([64], 16, True), ([64] * 16, 16, True), ([128] * 128, 16, True), ([2048] + [1] * 511, 16, True),
    ([8192] + [20] * 100, 16, True), ([1500] + [27] * 20, 8, True), ([256] + [1] * 128, 8, True),
    ([16], 16, False), ([16] * 16, 16, False), ([24] * 128, 8, False), ([64] + [1] * 64, 16, False), ([256] + [1] * 128, 16, False), ([256] + [1] * 511, 8, False),
    ([1024] + [1] * 511, 16, False), ([64] * 64 + [1] * 448, 8, False), ([128] * 16 + [1] * 112, 16, False), ([1] * 512, 16, False)])
def test_which_steps_of_the_delta_rule_run_in_chunks(lens, heads, chunked):
    """Steps that were measured in both forms: the faster one."""
    from nanovllm import mixops
    assert (mixops.delta_chunks(max(lens), 128) and mixops.delta_pays(sum(lens), len(lens), max(lens), 2 * heads)) == chunked


def test_workspace_of_a_ragged_step_is_bounded_by_its_tokens_and_sequences():
    """Whatever the lengths: a row of sixteen tokens each, and one a sequence; what a step of many sequences needs beyond a step of one is what the model declares."""
    from nanovllm import _native, mixops
    of = _native.load_mix().b200m_channel_delta_workspace_bytes
    row = of(0, 1, 16)
    for lens in ([8192] + [20] * 100, [1] * 512, [16384], [17] * 512):
        n = sum(lens)
        assert of(n, len(lens), 16) == (n // 16 + len(lens)) * row >= sum(-(-l // 16) for l in lens) * row
        assert of(n, len(lens), 16) - of(n, 1, 16) <= mixops.delta_scratch_bytes(16, len(lens))
    assert mixops.delta_scratch_bytes(64, 4096) == mixops.DELTA_WORKSPACE        # no step takes more than that at a time
    layer = ChannelDeltaMixer(16, dict(heads=2, kv_heads=1, dim=96, vdim=8, conv=4), 1e-6, torch.bfloat16, "cpu")
    assert layer.step_scratch_bytes(512) == 512 * of(0, 1, 2)
    for dim, dtype in ((64, torch.bfloat16), (96, torch.float32)):             # forms that take none
        assert ChannelDeltaMixer(16, dict(heads=2, kv_heads=1, dim=dim, vdim=8, conv=4), 1e-6, dtype, "cpu").step_scratch_bytes(512) == 0
