"""What a step keeps between its layers belongs to its sizes (no GPU)."""
import dataclasses

import torch

from blitz_scale_b200.models.hybrid import HybridRunner
from blitz_scale_b200.models.llama import StepMeta


def step(T):
    none = torch.zeros(64, dtype=torch.int32)
    return StepMeta(ids=none, pos=none, slot=none, page_indices=none, page_indptr=none, last_page_len=none, batch=T, num_tokens=T)


def test_a_step_that_gets_other_sizes():
    r = HybridRunner.__new__(HybridRunner)
    r._columns, r._proj = [({"a": (0, 3), "b": (3, 2)}, 5, 0)], torch.zeros(100)
    m = step(6)
    first, parts = r._projection(0, m)
    assert first.shape == (6, 5) and r._projection(0, m)[0] is first and parts["b"].shape == (6, 2)
    m.num_tokens = 4
    assert r._projection(0, m)[0].shape == (4, 5)
    assert r._projection(0, dataclasses.replace(m, num_tokens=7))[1]["a"].shape == (7, 3)
