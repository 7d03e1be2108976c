"""Decode steps of a few rows through ops.linear_rows, host side: which steps take them, and what they hand from layer to layer.  The ops are CPU stand-ins."""
import pytest
import torch

import test_model_glue_cpu as glue
from oracle.qwen3_ref import add_rmsnorm_ref, rmsnorm_ref, silu_mul_ref


class FewRowsOps(glue.CpuOps):
    rows_seen: list = []
    attention_pdl: list = []

    def linear_rows(self, x, w, norm_w=None, eps=0.0, add=None, silu=False, splits=1, pdl=False):
        self._count("linear_rows")
        self.rows_seen.append(x.shape[0])
        assert w.is_contiguous() and x.shape[1] == w.shape[1] and x.shape[1] % (64 * splits) == 0 and (norm_w is None or splits == 1)
        assert (add is None or norm_w is not None) and (not silu or norm_w is not None)
        residual = x
        if add is not None:
            x, residual = add_rmsnorm_ref(add, x, norm_w, eps)
        elif norm_w is not None:
            x = rmsnorm_ref(x, norm_w, eps)
        ks = x.shape[1] // splits
        y = torch.zeros(x.shape[0], w.shape[0])
        for s in range(splits):
            y = y + x[:, s * ks:(s + 1) * ks].float() @ w[:, s * ks:(s + 1) * ks].float().t()
        y = y.to(torch.bfloat16)
        return (silu_mul_ref(y) if silu else y), residual

    def paged_decode(self, *args, **kw):
        self.attention_pdl.append(self.pdl_off.depth == 0)
        return super().paged_decode(*args, **kw)

    def paged_decode_fused(self, *args, **kw):
        self.attention_pdl.append(self.pdl_off.depth == 0)
        return super().paged_decode_fused(*args, **kw)


def run(monkeypatch, env, fused_decode_max=None, heads=4):
    from nanovllm.utils.synthetic import PRESETS
    for name in ("B200_LINEAR", "B200_LINEAR_MAX_ROWS"):
        monkeypatch.delenv(name, raising=False)
    monkeypatch.setitem(PRESETS, "tiny-wide", dict(PRESETS["tiny"], hidden_size=512, num_attention_heads=heads))
    monkeypatch.setattr(glue, "CpuOps", FewRowsOps)
    monkeypatch.setattr(FewRowsOps, "rows_seen", [])
    monkeypatch.setattr(FewRowsOps, "attention_pdl", [])
    return glue.run_product_model(monkeypatch, "tiny-wide", env, fused_decode_max)


def close(got, want):
    for g, w in zip(got, want):                             # only the order of the sums differs from the oracle
        assert ((g.float() - w.float()).norm() / w.float().norm()).item() < 1e-2


def test_few_row_steps_are_the_oracles(monkeypatch):
    got, want, fake, model = run(monkeypatch, {})
    assert model.few_rows == 16 and fake.calls["linear_rows"] % (4 * len(model.layers) - 1) == 0 and max(FewRowsOps.rows_seen) <= 16
    close(got, want)


@pytest.mark.parametrize("most", [0, 2])
def test_the_row_limit_of_the_own_products_holds_for_few_rows(most, monkeypatch):
    """B200_LINEAR_MAX_ROWS: steps of more rows are the library's."""
    got, want, _, model = run(monkeypatch, {"B200_LINEAR_MAX_ROWS": str(most)})
    assert max(FewRowsOps.rows_seen, default=0) <= most
    close(got, want)


@pytest.mark.parametrize("heads,fused_max", [(4, None), (4, 0), (8, None)])
def test_attention_of_few_rows_starts_when_the_projection_has_ended(heads, fused_max, monkeypatch):
    """Both forms of the attention behind it: without the early-launch attribute."""
    got, want, fake, _ = run(monkeypatch, {}, fused_max, heads)
    assert fake.calls["linear_rows"] > 0 and FewRowsOps.attention_pdl and not any(FewRowsOps.attention_pdl)
    close(got, want)
