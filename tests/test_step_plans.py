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
    assert ask()
    many = lambda **k: ops.prefill_on_tcgen05(Q, 2048, _step(2048), heads, kv_heads, hd, 0.125, **k)
    assert many(window=4096) and many(sink=torch.zeros(heads)) and many(window=16) == (hd == 128)
    assert not ops.prefill_on_tcgen05(Q, 2048, _step(64), heads, kv_heads, hd, 0.125, window=16)
    assert ask(window=4096) == (hd == 128 or 300 * heads >= ops.TCGEN05_WINDOW_ROWS)


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
    assert _runs(monkeypatch, step(64, 8, 500, host_new=[8] * 8)) == 0 and _runs(monkeypatch, step(128, 8, 500, host_new=[16] * 8)) == 16
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


# us with 1, 2, 4 and 8 CTAs a sequence, measured; rooms of 32 heads of 64 on 8, 32 of 128, 64 of 64, 16 of 64, 24 of 128
ROOMS = {"32x64": (35, 35, 34, 34), "32x128": (16, 16, 15, 15), "64x64": (13, 13, 13, 12), "16x64": (92, 92, 92, 91), "24x128": (49, 49, 49, 49)}


@pytest.mark.parametrize("heads,n,context_class,window,times", [
    ("32x64", 15, 0, 0, [(22.5, 16.8, 12.7, 11.2)]), ("32x64", 16, 0, 0, [(22.6, 16.6, 12.6, 20.8)]), ("32x64", 33, 0, 0, [(22.8, 16.6, 12.9, 31.3)]),
    ("32x64", 34, 0, 0, [(22.7, 16.6, 22.2, 31.7)]), ("32x64", 74, 0, 0, [(22.7, 17.0, 34.5, 53.4)]),
    ("32x64", 40, 2, 0, [(338, 177.6, 127.9, 108.7)]), ("32x64", 76, 2, 0, [(342.3, 349.1, 192.2, 214.3)]), ("32x64", 148, 2, 0, [(345.1, 354.4, 320.2, 360)]),
    ("32x64", 148, 2, 1024, [(91.9, 101.5, 147.8, 208.2)]), ("32x64", 76, 0, 0, [(23.1, 32.5, 36.5, 63.2)]),
    ("32x128", 76, 0, 0, [(31.3, 43.4, 46.3, 74.3)]), ("32x128", 148, 0, 0, [(36.9, 50.6, 82.2, 136.4)]), ("64x64", 76, 0, 0, [(39.2, 53.2, 59.5, 101.5)]),
    ("32x128", 40, 2, 1024, [(175.1, 99.3, 78.8, 80.0)]), ("32x128", 76, 2, 0, [(456.4, 466.4, 374.2, 287.7)]),
    ("64x64", 40, 2, 1024, [(209.6, 117.4, 95.8, 94.2)]), ("64x64", 76, 2, 1024, [(212.7, 230.7, 144.9, 188.3)]), ("64x64", 148, 2, 1024, [(212.5, 232.6, 240.9, 317)]),
    ("16x64", 40, 2, 0, [(263.2, 88.2, 95.9, 84.5)]), ("16x64", 148, 2, 0, [(266.2, 175.5, 238.7, 279.8)]), ("24x128", 148, 2, 0, [(362.2, 264.6, 356.4, 404.9)])])
def test_ctas_a_sequence_of_single_tokens(monkeypatch, heads, n, context_class, window, times):
    monkeypatch.setattr(ops, "sm_count", lambda: 148)
    ranks, chunks = ops.mixed_token_ranks(n, context_class, window, 64, ROOMS[heads])
    total = [sum(t[i] for t in times) for i in range(4)]
    assert total[(1, 2, 4, 8).index(ranks)] <= 1.05 * min(total), (ranks, total)
    assert ranks * chunks >= (35 if window else 32 << context_class)


def test_recurrences_of_captured_steps_whose_rows_may_be_empty():
    """A prompt of a few tokens is 64 rows in a captured step: it is walked, as it is alone."""
    assert ops.delta_in_chunks(_step(96)) and not ops.delta_in_chunks(_step(95))
    assert not ops.delta_in_chunks(_step(128, captured=True)) and ops.delta_in_chunks(_step(192, captured=True))
    assert not ops.delta_in_chunks(_step(500, 8)) and ops.delta_in_chunks(_step(512, 8))
    for heads, per_row in ((16, True), (64, True), (32, False)):
        assert ops.outer_in_chunks(_step(64), heads, per_row) and not ops.outer_in_chunks(_step(63), heads, per_row)
        assert not ops.outer_in_chunks(_step(64, captured=True), heads, per_row) and ops.outer_in_chunks(_step(128, captured=True), heads, per_row)
    assert ops.outer_in_chunks(_step(64, captured=True), 64, False) and not ops.outer_in_chunks(_step(300, 8), 64, False)


def test_float32_rows_of_many_sequences(monkeypatch):
    """Short runs after long contexts go by rows, whatever the average; long runs beside a short one go together."""
    step = lambda starts, news: _step(sum(news), len(news), max_context=max(a + b for a, b in zip(starts, news)), host_starts=starts, host_new=news)
    assert ops.simt_runs(step([0, 0, 0, 629, 12, 0, 0, 0, 0, 6, 6], [21, 25, 1, 1, 45, 56, 15, 1, 17, 3, 8]), 5, 5, 64) == 0
    assert ops.simt_runs(step([500] * 8, [3] * 8), 32, 8, 64) == 0
    assert ops.simt_runs(step([600, 900, 500, 662], [145, 186, 4, 1]), 32, 8, 128) > 0
    assert ops.simt_runs(step([0, 30], [500, 300]), 32, 8, 64) == 400 and ops.simt_runs(step([0, 83, 0], [118, 27, 174]), 5, 5, 64) == 106
    assert ops.simt_runs(step([0, 224], [103, 23]), 5, 5, 64) == 0              # (16.4 us, 20.1 together)
    assert ops.simt_runs(step([0], [64]), 32, 8, 64) == 64 and ops.simt_runs(step([0], [3]), 32, 8, 64) == 0


@pytest.mark.parametrize("M,N,K,first", [(33, 640, 640, True), (48, 2048, 768, True), (33, 1536, 1024, False), (64, 2560, 1024, True), (64, 1024, 1024, False),
                                         (33, 3072, 2048, False), (64, 3072, 2048, False), (64, 6144, 2048, True), (32, 640, 640, False), (48, 2048, 4096, False)])
def test_products_of_33_to_64_tokens_take_the_faster_way_round(monkeypatch, M, N, K, first):
    monkeypatch.setattr(ops, "sm_count", lambda: 148)
    assert ops.tokens_first(M, N, K) == first
