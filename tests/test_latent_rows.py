"""Which form a latent prompt step takes and what it holds (mixops.latent_expands, latent_costs, latent_scratch_bytes): host arithmetic, no GPU."""
import pytest
import torch

from nanovllm import mixops as mx
from nanovllm.utils.context import get_context, reset_context, set_context


def step(len_q, len_k, heads=16, rank=512, bs=256, window=0, known=True, spare=0):
    """(rows, longest) and whether keys and values are formed; ``spare``: table columns beyond the longest sequence."""
    n, width = sum(len_q), -(-max(len_k) // bs) + spare
    q = torch.empty(n, heads, 192, dtype=torch.bfloat16)
    cache, tables = torch.empty(8, rank + 64, dtype=torch.bfloat16), torch.empty(len(len_q), width, dtype=torch.int32)
    cu = torch.empty(len(len_q) + 1, dtype=torch.int32)
    spans = mx.StepSpans(len(len_q), max(len_q), cu, cu, None, *((max(len_k), sum(len_k)) if known else ()))
    return mx._latent_rows(n, tables, bs, spans, window), mx.latent_expands(q, 128, 64, 128, rank, 0.07, cache, tables, bs, spans, window)


def test_rows_are_those_that_exist():
    """Ragged steps count their keys, not sequences times the widest table; without lengths on the host the tables bound them."""
    ragged = [100] * 31 + [4096]
    assert step(ragged, ragged) == ((31 * 100 + 4096, 4096), True)
    assert step(ragged, ragged, spare=100)[0] == (31 * 100 + 4096, 4096)
    assert step([64] * 33, [64] * 32 + [4096])[1]                        # a sequence more than 2^17 padded rows hold
    assert step([7, 9], [300, 600], known=False)[0] == (2 * 768, 768)
    assert step([2048] * 4, [2048] * 4) == ((8192, 2048), True)


def test_a_window_bounds_the_rows():
    (rows, most), formed = step([16], [30000], window=1024)
    assert rows == most == 1039 and formed
    assert step([16] * 8, [16000] * 8, window=512)[0] == (8 * 527, 527)
    assert step([600, 5], [600, 40], window=10_000)[0] == (640, 600)     # wider than every context


@pytest.mark.parametrize("heads,rank,seqs,q,k,formed", [
    (16, 512, 1, 4, 2048, True), (16, 512, 16, 4, 2048, True), (16, 512, 32, 4, 2048, False), (16, 512, 64, 4, 2048, False), (16, 512, 64, 32, 2048, True),
    (16, 512, 64, 8, 512, False), (16, 512, 64, 16, 512, True), (16, 512, 128, 4, 512, False), (16, 512, 16, 128, 8192, True), (16, 256, 64, 16, 512, False),
    (16, 256, 64, 32, 512, True), (16, 256, 16, 4, 8192, False), (16, 256, 1, 4, 8192, True), (4, 512, 16, 4, 2048, True), (4, 512, 64, 16, 2048, True)])
def test_the_faster_form_is_taken(heads, rank, seqs, q, k, formed):
    """Points of the measured table whose two times differ by more than a tenth."""
    assert step([q] * seqs, [k] * seqs, heads, rank)[1] is formed


def test_scratch_is_bounded_and_known():
    """What a step may hold grows with its rows up to a bound that does not grow with the heads, and a step beyond the bound takes the latents."""
    of = lambda rows, heads=16: mx.latent_scratch_bytes(heads, 128, 128, 576, rows)
    assert of(1000) == 1000 * (576 * 2 + 16 * 512)
    assert of(1 << 30) == of(1 << 40) == of(1 << 30, 128) == mx.LATENT_ROWS_BYTES + mx.LATENT_KV_BYTES
    most = mx.LATENT_ROWS_BYTES // (576 * 2)
    assert step([512], [most])[1] and not step([512], [most + 1])[1]


def test_context_carries_the_total():
    set_context(True, None, None, 3, 9, total_seqlen_k=21)
    assert get_context().total_seqlen_k == 21
    reset_context()
    assert get_context().total_seqlen_k == 0
