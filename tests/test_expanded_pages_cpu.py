"""Tables of a prompt's expanded pages belong to one pass (no GPU)."""
import types

import pytest
import torch

from blitz_scale_b200.models.hybrid import HybridRunner
from blitz_scale_b200.models.llama import StepMeta


@pytest.mark.parametrize("window", [0, 20])
def test_a_step_that_is_used_again(window):
    runner = HybridRunner.__new__(HybridRunner)
    runner.page_size, runner.runs = 16, [types.SimpleNamespace(layer=0)]
    runner.cfg = types.SimpleNamespace(streams=1, layer_specs=[None])
    runner._run_layer_streams = lambda *a: None
    none = torch.empty(0)
    m = StepMeta(ids=none, pos=none, slot=none, page_indices=torch.arange(40, dtype=torch.int32) + 7, page_indptr=none, last_page_len=none,
                 seq_lens_host=[30, 50], kv_lens_host=[30, 50], is_prefill=True, batch=2, num_tokens=80)
    ask = lambda: runner._expanded_pages(m, 0, window, torch.device("cpu"))
    runner.run_layer(0, m)
    first = ask()
    assert ask()[0] is first[0]                                  # once per pass
    m.kv_lens_host = [90, 200]                                   # the sequences have grown,
    m.page_indices.copy_(torch.arange(40, dtype=torch.int32).flip(0))    # and other pages hold them
    runner.run_layer(0, m)
    got, runner._expanded = ask(), None
    for a, b in zip(got, ask()):
        assert torch.equal(a, b) if isinstance(a, torch.Tensor) else a == b
