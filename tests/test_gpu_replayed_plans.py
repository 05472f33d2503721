"""A small step's graph is replayed for every step of as many sequences, rows and wanted places, wherever those stand: it gives what a graph gives that was
captured there."""
from __future__ import annotations

import pytest
import torch

import bededra_helpers
import dofevik_helpers

pytestmark = pytest.mark.gpu


def _bededra(folder):
    left = bededra_helpers._left(16, 4, 32, 32, 0.18, 20.0, 1024, 64)
    c = bededra_helpers._model(97, 256, 2, [dict(bededra_helpers._par(left, bededra_helpers._right(4, 64, 32, 16.0, 8), 1.0, 1.0), mlp=None)])
    bededra_helpers.write_folder(folder, c, bededra_helpers.random_weights(c, 3))
    return c


def _dofevik(folder):
    c = dofevik_helpers._model(97, 256, [dict(dofevik_helpers._att(16, 4, 64, 64, 0.125, 1024, 10000.0, 32), mlp=None),
                                         dict(dofevik_helpers._att(8, 8, 64, 64, 0.125, 2048, 10000.0, 32), mlp=None)])
    dofevik_helpers.write_folder(folder, c, dofevik_helpers.random_weights(c, 3))
    return c


def _replayed_and_fresh(folder, vocab, portion, before, capture_at):
    """Logits of a portion behind ``before`` tokens: from a graph that was captured ``capture_at`` tokens in, and from one captured there."""
    from kuiperllama_b200.engine import Engine, SequenceInput, load_model
    with torch.inference_mode():
        model = load_model(folder, dtype="bfloat16", device="cuda:0")
        out = []
        for first in (capture_at, None):
            eng = Engine(model, model.new_cache(max_tokens=64 * 80), use_graphs=True)
            feed = lambda slot, toks, want: eng.step([SequenceInput(slot, toks, want)])
            toks = lambda n, seed: bededra_helpers.tokens(n, vocab, seed=seed)
            if first is not None:
                slot = eng.alloc_slot()
                if first:
                    feed(slot, toks(first, 9), [])
                feed(slot, toks(portion, 8), list(range(portion)))
                eng.free_slot(slot)
            slot = eng.alloc_slot()
            if before:
                feed(slot, toks(before, 1), [])
            out.append(feed(slot, toks(portion, 2), list(range(portion))).clone())
            assert len(eng._step_graphs) == 1
            eng.check_device_errors()
    return out


@pytest.mark.parametrize("portion,before,capture_at", [(64, 1500, 0), (64, 0, 1500), (200, 1500, 0)])
def test_mixed_heads_of_a_replayed_portion(tmp_path, portion, before, capture_at):
    c = _bededra(str(tmp_path))
    replayed, fresh = _replayed_and_fresh(str(tmp_path), c["vocab"], portion, before, capture_at)
    assert torch.equal(replayed, fresh)


@pytest.mark.parametrize("portion,before,capture_at", [(64, 1500, 0), (300, 1500, 0), (512, 0, 1500)])
def test_windows_of_a_replayed_portion(tmp_path, portion, before, capture_at):
    c = _dofevik(str(tmp_path))
    replayed, fresh = _replayed_and_fresh(str(tmp_path), c["vocab"], portion, before, capture_at)
    assert torch.equal(replayed, fresh)
