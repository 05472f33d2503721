"""How a launch is planned from what a step says: steps that say less than the engine's are taken, and what a captured step is replayed for does not
depend on where its sequences stood when it was captured."""
from __future__ import annotations

from types import SimpleNamespace

import pytest
import torch

from kuiperllama_b200.csrc import ops

Q = torch.zeros(64, 64 * 32, dtype=torch.bfloat16)


def _step(rows, seqs=1, **more):
    return SimpleNamespace(n_tokens=rows, n_seqs=seqs, max_new=rows, is_decode=False, **more)


@pytest.mark.parametrize("heads,kv_heads,hd", [(32, 8, 64), (16, 16, 64), (8, 2, 128)])
def test_prompts_without_a_context_choose_a_kernel(heads, kv_heads, hd):
    ask = lambda **k: ops.prefill_on_tcgen05(Q, 2048, _step(300), heads, kv_heads, hd, 0.125, **k)
    assert ask() and ask(window=4096) and ask(sink=torch.zeros(heads))
    assert ask(window=16) == (hd == 128)


@pytest.mark.parametrize("heads,kv_heads", [(32, 8), (16, 16)])
@pytest.mark.parametrize("window", [0, 16, 512, 1024, 4096])
@pytest.mark.parametrize("rows", [64, 256, 512])
def test_a_captured_step_chooses_by_what_its_replays_share(heads, kv_heads, window, rows):
    sink = None if window else torch.zeros(heads)
    chosen = {ops.prefill_on_tcgen05(Q, 2048, _step(rows, captured=True, max_context=n), heads, kv_heads, 64, 0.125, window, sink) for n in (1, 300, 600, 5000)}
    assert len(chosen) == 1


@pytest.mark.parametrize("rows,seqs", [(5, 1), (64, 1), (64, 8), (150, 1), (512, 3), (2048, 1), (100000, 7)])
def test_pieces_of_mixed_heads_follow_from_rows_and_sequences(rows, seqs):
    s0, s1 = ops.mixed_prompt_splits(_step(rows, seqs))
    assert 1 <= s1 <= s0 <= 16 and s0 <= 2 * s1
    assert s1 == 1 or s1 * (rows // 8 + seqs) < 300 + rows // 8 + seqs


def _runs(monkeypatch, step):
    asked = []
    monkeypatch.setattr(ops, "attention_simt", lambda *a, **k: asked.append(k["runs"]))
    q = torch.zeros(step.n_tokens, 64)
    ops.attention(q, 64, q, None, None, None, step, 1, 1, 64, 0.125)
    return asked[0]


def test_rows_that_float32_attention_takes_together(monkeypatch):
    places = dict(positions=None, token_slot=None)
    step = lambda rows, seqs, context, **more: _step(rows, seqs, max_context=context, **places, **more)
    assert _runs(monkeypatch, step(64, 1, 64)) == 64                                     # (no word of what each sequence brings)
    assert _runs(monkeypatch, step(24, 8, 500)) == 0 and _runs(monkeypatch, step(24, 8, 500, host_new=[3] * 8)) == 0
    assert _runs(monkeypatch, step(64, 8, 500, host_new=[8] * 8)) == 8
    assert _runs(monkeypatch, step(64, 2, 100, host_new=[63, 1])) == 0 and _runs(monkeypatch, step(64, 2, 500, host_new=[63, 1])) == 32
    for rows, seqs in ((64, 1), (64, 8), (512, 8), (128, 2)):
        seen = {_runs(monkeypatch, step(rows, seqs, context, captured=True, host_new=news))
                for context in (rows, 3000) for news in ([rows // seqs] * seqs, [rows - seqs + 1] + [1] * (seqs - 1))}
        assert len(seen) == 1, (rows, seqs, seen)


@pytest.mark.parametrize("N,K", [(4096, 4096), (4096, 14336), (4096, 11008), (5120, 5120), (2048, 8192), (3072, 2048), (6144, 4096), (2560, 2560)])
@pytest.mark.parametrize("M", [1, 4, 8, 16])
def test_products_of_few_tokens_have_a_cta_for_every_sm(monkeypatch, N, K, M):
    monkeypatch.setattr(ops, "sm_count", lambda: 148)
    pieces = ops.skinny_splits(N, K, M)
    assert 148 < pieces * -(-N // 128) <= 296 or pieces == 8 or pieces == -(-K // 64) // 4
    assert pieces <= 8
