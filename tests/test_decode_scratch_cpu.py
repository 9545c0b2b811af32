"""Scratch of decode attention whose address captured graphs hold, by the runner's own bookkeeping (no GPU)."""
import weakref

import pytest
import torch

from blitz_scale_b200 import ops
from blitz_scale_b200.models.config import get_config
from blitz_scale_b200.models.llama import LlamaRunner
from blitz_scale_b200.models.weights import WeightSegment


@pytest.mark.parametrize("first,then", [((1, 16), (2, 16)), ((2, 16), (9, 4)), ((4, 0), (200, 0))])
def test_scratch_outlives_a_larger_one(monkeypatch, first, then):
    monkeypatch.setattr(ops, "attn_decode_workspace_bytes", lambda B, heads, dim, splits: B * heads * max(1, splits) * (dim + 1) * 4)
    cfg = get_config("tiny_gpu")
    kv = torch.zeros(cfg.layers, 2, 2, 16, cfg.kv_heads, cfg.head_dim, dtype=torch.bfloat16)
    runner = LlamaRunner(WeightSegment(cfg, 1, 0, torch.bfloat16, device="cpu"), kv, 256, 256)
    address = runner._workspace(*first).data_ptr()
    alive = weakref.ref(runner._workspace(*first))
    grown = runner._workspace(*then)
    assert grown.data_ptr() != address and runner._workspace(*then) is grown
    assert alive() is not None and alive().data_ptr() == address
