"""Whole decode steps through the row-wise products of a few rows (``_forward_few_rows``) against the same steps on the launches they replace, bit for bit: the residual
handed from layer to layer, the projection that the next layer adds, the last layer's partial sums.  Sizes are the benchmark model's, with few layers."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layers,heads,kv_heads,fused_max", [(1, 16, 8, None), (3, 16, 8, None), (2, 16, 8, 0), (2, 16, 4, None)])
def test_same_logits_as_the_launches_replaced(layers, heads, kv_heads, fused_max, monkeypatch):
    from nanovllm import ops
    from nanovllm.models.qwen3 import Qwen3ForCausalLM
    from nanovllm.utils.context import reset_context, set_context
    from nanovllm.utils.synthetic import PRESETS, hf_config_dict, random_weights
    for name in ("B200_LINEAR", "B200_LINEAR_MAX_ROWS", "B200_LINEAR_CFG"):
        monkeypatch.delenv(name, raising=False)
    dims = dict(PRESETS["qwen3-0.6b"], num_hidden_layers=layers, num_attention_heads=heads, num_key_value_heads=kv_heads, vocab_size=2048)
    model = Qwen3ForCausalLM(SimpleNamespace(**hf_config_dict(dims)), 0, 1, "cuda", max_position=4096)
    for name, w in random_weights(dims, seed=3).items():
        model.load_hf_tensor(name, w)
    if fused_max is not None:
        model.fused_decode_max_batch = fused_max
    assert model.few_rows == 16
    bs, per = 16, 6
    start = torch.randn(ops.kv_cache_shape(layers, 17 * per, kv_heads, bs, 128), device="cuda", generator=torch.Generator(device="cuda").manual_seed(4)).bfloat16()
    kv = start.clone()
    ops.bind_kv_cache(kv)
    for i, a in enumerate(model.modules()):
        a.k_cache, a.v_cache, a.layer_id = kv[0, i], kv[1, i], i
    for rows in (1, 8, 9, 16, 17):
        lens = [1 + (i * 7) % (bs * per) for i in range(rows)]
        tables = [list(range(i * per, (i + 1) * per)) for i in range(rows)]
        i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
        ids = torch.randint(0, 2048, (rows,), device="cuda", generator=torch.Generator(device="cuda").manual_seed(rows))
        pos = torch.tensor([l - 1 for l in lens], dtype=torch.int64, device="cuda")
        got = []
        for few in (16, 0):
            model.few_rows = few
            kv.copy_(start)
            set_context(False, slot_mapping=i32([t[(l - 1) // bs] * bs + (l - 1) % bs for t, l in zip(tables, lens)]), context_lens=i32(lens), block_tables=i32(tables))
            got.append((model.compute_logits(model(ids, pos)), kv.clone()))
            reset_context()
        assert torch.isfinite(got[0][0]).all() and torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1]), rows
