"""What a prompt's results owe to the way it is cut into steps: in 32-bit arithmetic nothing, to the last bit."""
from __future__ import annotations

import pytest
import torch

from bededra_helpers import CONFIGS, random_weights, tokens, write_folder

pytestmark = pytest.mark.gpu


def _logits(model, toks, cuts):
    from kuiperllama_b200.engine import Engine, SequenceInput
    eng, rows, at = Engine(model, model.new_cache(max_tokens=64 * 16)), [], 0
    with torch.inference_mode():
        slot = eng.alloc_slot()
        for n in cuts:
            rows.append(eng.step([SequenceInput(slot, toks[at:at + n], list(range(n)))]).clone())
            at += n
        eng.free_slot(slot)
    eng.check_device_errors()
    return torch.cat(rows)


@pytest.mark.parametrize("name", ["wide", "mixed", "odd"])
def test_float32_prompts_have_the_same_bits_however_they_are_cut(tmp_path, name):
    """State-space layers, linear attention and mixed heads: steps of 9 tokens and more, on both sides of where bfloat16 models work in chunks."""
    from kuiperllama_b200.engine import load_model
    c = CONFIGS[name]
    folder = write_folder(str(tmp_path), c, random_weights(c, 1))
    toks = tokens(330, c["vocab"], seed=4)
    with torch.inference_mode():
        model = load_model(folder, dtype="float32", device="cuda:0")
    whole = _logits(model, toks, [330])
    for cuts in ([330], [300, 30], [31, 299], [63, 64, 65, 96, 42], [9] * 30 + [60]):
        got = _logits(model, toks, cuts)
        assert torch.equal(whole, got), (cuts, int((whole != got).any(dim=1).nonzero()[0]))


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("kernel", ["chunked", "walk"])
def test_a_recurrence_is_walked_in_float32_and_where_its_part_says_so(monkeypatch, tmp_path, dtype, kernel):
    import terolix_helpers
    from kuiperllama_b200.csrc import ops
    from kuiperllama_b200.engine import load_model
    from kuiperllama_b200.parts import GatedDeltaMixer, GatedLinearAttentionMixer, Mamba2Mixer
    asked = []

    def listen(name):
        real = getattr(ops, name)
        monkeypatch.setattr(ops, name, lambda *a, **k: (asked.append((name, k["chunked"])), real(*a, **k))[1])

    for name in ("outer_recurrence", "gated_delta_rule"):
        listen(name)
    for part in (GatedDeltaMixer, GatedLinearAttentionMixer, Mamba2Mixer):
        monkeypatch.setattr(part, "KERNEL", kernel)
    b, t = CONFIGS["wide"], terolix_helpers.CONFIGS["mixed"]
    (tmp_path / "b").mkdir(), (tmp_path / "t").mkdir()
    folders = (write_folder(str(tmp_path / "b"), b, random_weights(b, 1)), str(tmp_path / "t"))
    terolix_helpers.write_folder(folders[1], t, terolix_helpers.random_weights(t, seed=1))
    for folder, c in zip(folders, (b, t)):
        with torch.inference_mode():
            model = load_model(folder, dtype=dtype, device="cuda:0")
        assert bool(torch.isfinite(_logits(model, tokens(130, c["vocab"], seed=4), [130])).all())
    assert {n for n, _ in asked} == {"outer_recurrence", "gated_delta_rule"}
    assert {c for _, c in asked} == {None if dtype == "bfloat16" and kernel == "chunked" else False}
