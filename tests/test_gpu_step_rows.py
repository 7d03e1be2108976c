"""Whole decode steps as one kernel (csrc/step_rows.cu) against the launches it replaces (``_forward_few_rows``), bit for bit: hidden states and cache.  Rows on both sides of
the ways the norms are split over warps, one and two query heads per kv head, every number of ring slots of the narrow products, one and two column halves of the
residual, contexts of nothing but the step's own token, padding rows, page edges, contexts over one CTA and over eight."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu


def build(monkeypatch, layers, hidden, inter, heads, kv_heads, pages, block, positions=4096):
    from nanovllm import ops
    from nanovllm.models.qwen3 import Qwen3ForCausalLM
    from nanovllm.utils.synthetic import PRESETS, hf_config_dict, random_weights
    for name in ("B200_LINEAR", "B200_LINEAR_MAX_ROWS", "B200_LINEAR_CFG", "B200_FUSED_DECODE_MAX"):
        monkeypatch.delenv(name, raising=False)
    dims = dict(PRESETS["qwen3-0.6b"], num_hidden_layers=layers, hidden_size=hidden, intermediate_size=inter, num_attention_heads=heads, num_key_value_heads=kv_heads,
                vocab_size=512)
    model = Qwen3ForCausalLM(SimpleNamespace(**hf_config_dict(dims)), 0, 1, "cuda", max_position=positions)
    for name, w in random_weights(dims, seed=5).items():
        model.load_hf_tensor(name, w)
    start = torch.randn(ops.kv_cache_shape(layers, pages, kv_heads, block, 128), device="cuda", generator=torch.Generator(device="cuda").manual_seed(6)).bfloat16()
    kv = start.clone()
    ops.bind_kv_cache(kv)
    for i, a in enumerate(model.modules()):
        a.k_cache, a.v_cache, a.layer_id = kv[0, i], kv[1, i], i
    return model, kv, start


def i32(v):
    return torch.tensor(v, dtype=torch.int32, device="cuda")


def step(model, kv, start, lens, tables, ids, one, capture=False):
    from nanovllm.utils.context import reset_context, set_context
    model.one_kernel_step = one
    context = dict(slot_mapping=None, context_lens=i32(lens), block_tables=i32(tables))
    pos = torch.tensor([max(l - 1, 0) for l in lens], dtype=torch.int64, device="cuda")

    def run():
        set_context(False, **context)
        out = model(ids, pos)
        reset_context()
        return out

    kv.copy_(start)
    if not capture:
        return run(), kv.clone()
    run()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = run()
    kv.copy_(start)
    graph.replay()
    graph.replay()                                          # the same step again: nothing is left over from the first
    return out.clone(), kv.clone()


@pytest.mark.parametrize("hidden,inter,heads,kv_heads", [(1024, 3072, 16, 8), (512, 1024, 8, 8), (1024, 2048, 24, 12), (512, 3072, 8, 4)])
@pytest.mark.parametrize("block,per", [(16, 20), (256, 4)])
def test_same_bits_as_the_launches_replaced(hidden, inter, heads, kv_heads, block, per, monkeypatch):
    from nanovllm import ops
    model, kv, start = build(monkeypatch, 3, hidden, inter, heads, kv_heads, 8 * per, block)
    most = block * per
    calls = []
    real = ops.step_rows
    monkeypatch.setattr(ops, "step_rows", lambda *a: calls.append(real(*a)) or calls[-1])
    for rows in (1, 2, 3, 4, 5, 8):
        lens = [[1, 0, 17, most, 16, block + 1, most - 1, 2][(i + rows) % 8] for i in range(rows)]
        tables = torch.randperm(8 * per, generator=torch.Generator().manual_seed(rows)).view(8, per)[:rows].tolist()
        ids = torch.randint(-1, 513, (rows,), device="cuda", generator=torch.Generator(device="cuda").manual_seed(rows))
        want = step(model, kv, start, lens, tables, ids, False)
        for capture in (False, True):
            del calls[:]
            got = step(model, kv, start, lens, tables, ids, True, capture)
            assert calls and all(c is not None for c in calls)
            assert torch.isfinite(got[0]).all() and torch.equal(got[0], want[0]) and torch.equal(got[1], want[1]), (rows, capture)


@pytest.mark.parametrize("hidden,inter,heads,kv_heads", [(1024, 1024, 16, 8), (512, 1024, 8, 8), (1024, 1024, 24, 12)])
@pytest.mark.parametrize("rows,block", [(1, 16), (1, 256), (2, 256), (3, 64), (4, 16), (8, 256)])
def test_contexts_up_to_the_rules_upper_end(rows, block, hidden, inter, heads, kv_heads, monkeypatch):
    """Tables of the widest context that a step of this kind may have, sixteen chunks of sixteen tokens a warp: contexts that fill them and that end around a turn of a CTA's warps, rows of
    any length beside them.  One page more, and the step is the launches'."""
    from nanovllm import ops
    from nanovllm import _native as nat
    splits = 1
    while splits < 8 and rows * kv_heads * splits * 2 <= nat.handle().sm_count:
        splits *= 2
    most = 16 * 16 * 8 * splits
    per = most // block
    model, kv, start = build(monkeypatch, 2, hidden, inter, heads, kv_heads, rows * per, block, most)
    calls = []
    real = ops.step_rows
    monkeypatch.setattr(ops, "step_rows", lambda *a: calls.append(real(*a)) or calls[-1])
    ids = torch.arange(rows, device="cuda")
    for turn, first in enumerate((most, most // 2 + 1, most // 8 * 3)):
        lens = [[first, 5, most - 128, most // 16, 128 * splits + 1, most - 1, 1, most // 3][i] for i in range(rows)]
        tables = torch.randperm(rows * per, generator=torch.Generator().manual_seed(turn)).view(rows, per)
        for i, l in enumerate(lens):
            tables[i, -(-l // block):] = -1                     # as the engine leaves them
        want = step(model, kv, start, lens, tables.tolist(), ids, False)
        del calls[:]
        got = step(model, kv, start, lens, tables.tolist(), ids, True)
        assert len(calls) == 1 and calls[0] is not None
        assert torch.isfinite(got[0]).all() and torch.equal(got[0], want[0]) and torch.equal(got[1], want[1]), lens
    h = nat.handle()
    need = lambda width: h.lib.b200_step_rows_workspace_bytes(h.ptr, rows, 2, hidden, inter, heads, width)
    assert need(per) > 0 and need(per + 1) == 0


@pytest.mark.parametrize("rows,hidden,inter,heads,kv_heads,per,asks", [(9, 1024, 3072, 16, 8, 4, True), (1, 1536, 1024, 8, 4, 4, True), (4, 1024, 1536, 16, 8, 4, True),
                                                                      (4, 1024, 1024, 12, 6, 4, True), (4, 1024, 1024, 16, 4, 4, False), (8, 1024, 1024, 16, 8, 400, True)])
def test_other_steps_keep_their_launches(rows, hidden, inter, heads, kv_heads, per, asks, monkeypatch):
    """More rows, other widths, wider head groups (which the model itself keeps from asking), contexts too long for the kernel: it refuses the step, and the others take it."""
    from nanovllm import ops
    from nanovllm import _native as nat
    model, kv, start = build(monkeypatch, 1, hidden, inter, heads, kv_heads, 16, 16)
    calls = []
    real = ops.step_rows
    monkeypatch.setattr(ops, "step_rows", lambda *a: calls.append(real(*a)) or calls[-1])
    ids = torch.arange(rows, device="cuda")
    lens, tables = [16] * rows, [[i] + [-1] * (per - 1) for i in range(rows)]
    want = step(model, kv, start, lens, tables, ids, False)
    assert not calls
    out, cache = step(model, kv, start, lens, tables, ids, True)
    assert bool(calls) == asks and all(c is None for c in calls)
    assert torch.isfinite(out).all() and torch.equal(out, want[0]) and torch.equal(cache, want[1])
    h = nat.handle()
    assert h.lib.b200_step_rows_workspace_bytes(h.ptr, rows, 1, hidden, inter, heads, per) == 0
    L = model.layers[0]
    assert real(ids, model.embed, [(L.qkv, L.o, L.gate_up, L.down, L.ln1, L.ln2, L.q_norm, L.k_norm)], model.norm, model.eps, model.cos_sin, i32(tables), i32(lens), heads,
                model.attn[0].scale) is None


def test_two_streams_have_a_workspace_each(monkeypatch):
    model, kv, start = build(monkeypatch, 2, 1024, 1024, 16, 8, 16, 16)
    ids = [torch.tensor([3, 4], device="cuda"), torch.tensor([5, 6], device="cuda")]
    tables = [[[0, 1], [2, 3]], [[4, 5], [6, 7]]]
    want = [step(model, kv, start, [20, 31], t, i, False)[0] for t, i in zip(tables, ids)]
    kv.copy_(start)
    from nanovllm.utils.context import reset_context, set_context
    model.one_kernel_step = True
    pos = torch.tensor([19, 30], device="cuda")
    lens, tabs = i32([20, 31]), [i32(t) for t in tables]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    got = [[], []]
    for _ in range(8):
        for k, s in enumerate(streams):
            with torch.cuda.stream(s):
                set_context(False, slot_mapping=None, context_lens=lens, block_tables=tabs[k])
                got[k].append(model(ids[k], pos))
                reset_context()
    torch.cuda.synchronize()
    assert all(torch.equal(o, want[k]) for k in (0, 1) for o in got[k])
