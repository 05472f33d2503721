"""The wanted places of a step: checked as one array, with the answers that one by one gave."""
from __future__ import annotations

import os
import sysconfig

import numpy as np
import pytest


@pytest.mark.parametrize("want", [[0], [3, 1, 1], (4,), range(5), range(4, -1, -2), range(0), np.array([2, 0]), [np.int64(4)]])
def test_places_are_taken(want):
    from kuiperllama_b200.engine.step import _places
    got = _places(want, 5, 0)
    assert got.dtype == np.int32 and got.tolist() == [int(w) for w in want]


@pytest.mark.parametrize("want,first", [([5], 5), ([0, -1, 9], -1), (range(6), 5), (range(-1, 3), -1), ([10 ** 30], 10 ** 30), (np.array([7]), 7),
                                        ([0.0, float("nan")], float("nan"))])
def test_places_outside_are_refused(want, first):
    from kuiperllama_b200.engine.step import StepError, _places
    with pytest.raises(StepError, match=f"slot 3: wanted place {first} is outside its 5 tokens"):
        _places(want, 5, 3)


@pytest.mark.parametrize("want", [{0, 2}, {1: 0}, [[0], [1]], [[0, 1]], ["1"], [None]])
def test_what_is_no_sequence_of_places_is_refused(want):
    from kuiperllama_b200.engine.step import _places
    with pytest.raises(TypeError):
        _places(want, 5, 3)


@pytest.mark.parametrize("tokens", [[5], [3, 0, 127999, 2], (7, 8), [-1, 4], [2 ** 31, 1], [-2 ** 40, 2 ** 40], [True, 2], [1.5, 2], range(4), np.array([3, 9]),
                                    np.array([4, 5], dtype=np.int32), [np.int64(6), 7], [2 ** 63, 0], ["a", 1], [[1], [2]], [None]])
def test_token_ids_are_what_numpy_makes_of_them(tokens):
    """Lists and tuples of plain ints take a routine of their own; everything else, and every refusal, is numpy's."""
    from kuiperllama_b200.engine import step

    def by_numpy():
        a = np.asarray(tokens, dtype=np.int64)
        return a.astype(np.int32), int(a.min()), int(a.max())

    try:
        want = by_numpy()
    except Exception as e:
        with pytest.raises(type(e)):
            step._token_ids(tokens, len(tokens))
        return
    got = step._token_ids(tokens, len(tokens))
    assert got[0].dtype == np.int32 and np.array_equal(got[0], want[0]) and got[1:] == want[1:]


def test_token_ids_of_a_long_prompt():
    from kuiperllama_b200.engine import step
    tokens = [(i * 7919) % 128256 for i in range(5000)]
    ids, lo, hi = step._token_ids(tokens, len(tokens))
    assert ids.tolist() == tokens and (lo, hi) == (min(tokens), max(tokens))
    assert step._host_tokens or not os.path.exists(os.path.join(sysconfig.get_paths()["include"], "Python.h"))


def test_a_build_without_the_interpreters_headers_leaves_out_what_needs_them(monkeypatch):
    """Everything else is built, a failure of anything else is one, and ids go through numpy."""
    from kuiperllama_b200.csrc import build
    from kuiperllama_b200.engine import step

    def fails(*names):
        def ensure_built(name, quiet=False):
            if name in names:
                raise build.ExtensionError(f"nvcc failed on {name}")
            return f"{name}.so"
        return ensure_built

    monkeypatch.setattr(build, "ensure_built", fails("host_tokens"))
    assert build.build_all(quiet=True) == {n: f"{n}.so" for n in build.SOURCES if n != "host_tokens"}
    monkeypatch.setattr(step, "_host_tokens", None)
    ids, lo, hi = step._token_ids([5, 2, 9], 3)
    assert ids.tolist() == [5, 2, 9] and (lo, hi) == (2, 9) and step._host_tokens is False
    monkeypatch.setattr(build, "ensure_built", fails("norms"))
    with pytest.raises(build.ExtensionError):
        build.build_all(quiet=True)
