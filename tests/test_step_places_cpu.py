"""Places that a step is asked for beyond its requests are refused before anything runs (no GPU)."""
import types

import pytest
import torch

from blitz_scale_b200.runtime import engine as E


@pytest.mark.parametrize("want", [[[0], [0], [0]], [[], [], [1, 0]]])
def test_places_of_a_request_that_is_not_there(want):
    eng = E.Engine.__new__(E.Engine)
    eng.cfg, eng.tp, eng.max_batch, eng.max_batch_tokens, eng.device = types.SimpleNamespace(vocab=8), 1, 4, 64, torch.device("cpu")
    eng.status, passes = types.SimpleNamespace(fully_loaded=lambda: True), []
    eng._step_pass = lambda batch, counts, src: passes.append(src)
    with pytest.raises(IndexError):
        eng.step(types.SimpleNamespace(size=2), [1, 3], want)
    assert not passes
    eng.step(types.SimpleNamespace(size=2), [1, 3], [[0], [2]])
    assert passes == [[(0, 0), (1, 2)]]
