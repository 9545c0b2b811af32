"""Who may say that a step's positions are in place before its pass starts (no GPU)."""
import types

import pytest
import torch

from blitz_scale_b200.models import llama
from blitz_scale_b200.models.llama import LlamaRunner, StepMeta


def step(T, **kw):
    none = torch.zeros(64, dtype=torch.int32)
    return StepMeta(ids=none, pos=none, slot=none, page_indices=none, page_indptr=none, last_page_len=none, batch=T, num_tokens=T, **kw)


class Ops:
    """Records what the kernels are called with."""
    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        return lambda *a, **kw: self.calls.append((name, a, kw))


@pytest.mark.parametrize("promised", [False, True])
def test_the_runner_promises_what_the_step_does(monkeypatch, promised):
    rec = Ops()
    monkeypatch.setattr(llama, "ops", rec)
    r = LlamaRunner.__new__(LlamaRunner)
    r.cfg = types.SimpleNamespace(rms_eps=1e-5, rope_theta=1e4)
    r.res = r.normed = r.qkv = r.attn = torch.zeros(8, 4)
    r.kv, r.qh, r.kvh, r.hd, r.page_size, r.tp = [None], 1, 1, 4, 16, 1
    r._w = lambda l, n: None
    r._workspace = lambda *a: None
    r.attention_block(0, step(3, **(dict(static_positions=True) if promised else {})))
    asked = [kw for name, _, kw in rec.calls if name == "rope_kv_store"]
    assert len(asked) == 1 and asked[0]["static_meta"] is promised


def test_engine_steps_promise():
    """The engine and the builder of steps bring positions by a copy."""
    from blitz_scale_b200.runtime.engine import Engine
    from blitz_scale_b200.runtime.meta import MetaBuilder
    eng = Engine.__new__(Engine)
    eng.layout = types.SimpleNamespace(ids=0, pos=8, slot=16, page_indices=24, page_indptr=32, last_page_len=48, tok_indptr=56, seq_slot=40)
    eng.dev = torch.zeros(64, dtype=torch.int32)
    assert eng._views(2, 2, 2, False).static_positions
    b = MetaBuilder(max_tokens=32, max_batch=4, max_pages_per_step=16, page_size=4, device="cpu")
    assert b.prefill([[1, 2, 3]], [[0, 1]]).static_positions and b.decode([5], [3], [[0, 1]]).static_positions
