"""Ragged steps of the chunked delta rule: one long portion among many short ones, empty ones and single tokens; more portions than the search for a workspace row looks
at together (128); a workspace of all chunks, of a few and of one.  Each against the form on the fp32 pipe, and the cut ones against the whole, bit for bit (a cut only sends the
state through memory)."""
import random

import pytest
import torch

from test_gpu_channel_delta import F64, inputs, rel, run

pytestmark = pytest.mark.gpu


def portions(kind):
    r = random.Random(3)
    return {"one long": [2] * 9 + [400] + [1] * 140, "empty": [0, 33, 0, 0, 17, 16, 0, 1, 0], "tiles": [16, 32, 15, 17, 31, 1, 48], "alone": [257],
            "many": [r.choice([0, 1, 15, 16, 17, r.randint(1, 70)]) for _ in range(300)]}[kind]


@pytest.mark.parametrize("kind", ["one long", "empty", "tiles", "alone", "many"])
def test_ragged_steps(kind, monkeypatch):
    from nanovllm import _native as nat, mixops as mx, ops
    lens = portions(kind)
    H, G, D, V = 2, 1, 128, 72
    a = inputs(lens, H, G, D, V, 7, -3.0)
    hist = [i % 3 == 0 and l > 0 for i, l in enumerate(lens)]
    monkeypatch.setattr(mx, "delta_pays", lambda *a: True)
    want, wstate = run(a, lens, hist, H, G, D, V, 1.0, forgetting=False)
    rows = sum(lens) // 16 + len(lens)
    row = nat.load_mix().b200m_channel_delta_workspace_bytes(0, 1, H)
    assert nat.load_mix().b200m_channel_delta_workspace_bytes(sum(lens), len(lens), H) == rows * row
    whole = None
    for fit in (rows, 7, 1) if rows < 60 else (rows, rows - 1, 23):
        monkeypatch.setattr(mx, "DELTA_WORKSPACE", fit * row + row - 1)
        before = ops.LAUNCHES[0]
        got, state = run(a, lens, hist, H, G, D, V, 1.0)
        assert ops.LAUNCHES[0] - before == 2 * -(-rows // min(fit, rows))
        assert rel(got, want.to(F64)) < 2e-6 and rel(state, wstate.to(F64)) < 2e-6
        assert torch.equal(state[[i for i, l in enumerate(lens) if l == 0]], wstate[[i for i, l in enumerate(lens) if l == 0]])
        whole = whole or (got, state)
        assert torch.equal(got, whole[0]) and torch.equal(state, whole[1])
