"""The wanted places of a step: checked as one array, with the answers that one by one gave."""
from __future__ import annotations

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
