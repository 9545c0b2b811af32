"""What a step keeps between its layers belongs to its sizes (no GPU)."""
import dataclasses
import types

import torch

from blitz_scale_b200.models import llama
from blitz_scale_b200.models.hybrid import HybridRunner
from blitz_scale_b200.models.llama import LlamaRunner, StepMeta


def step(T):
    none = torch.zeros(64, dtype=torch.int32)
    return StepMeta(ids=none, pos=none, slot=none, page_indices=none, page_indptr=none, last_page_len=none, batch=T, num_tokens=T)


def test_a_runner_that_gets_another_cache(monkeypatch):
    used = []
    fake = types.SimpleNamespace(rope_kv_store=lambda *a, **kw: used.append(a[3]), attn_decode=lambda *a, **kw: used.append(a[1]),
                                 rms_norm=lambda *a, **kw: None, gemm=lambda *a, **kw: None)
    monkeypatch.setattr(llama, "ops", fake)
    first, second = torch.zeros(2, 5, 2, 4, 1, 4), torch.ones(2, 5, 2, 4, 1, 4)
    cfg = types.SimpleNamespace(rms_eps=1e-5, rope_theta=1e4, layers=2, q_heads=1, kv_heads=1, head_dim=4, inter=8, hidden=4, vocab=16)
    seg = types.SimpleNamespace(cfg=cfg, tp=1, dtype=torch.float32, device="cpu", buffer=torch.zeros(1))
    r = LlamaRunner(seg, first, 8, 8)
    r._w, r._workspace = lambda l, n: None, lambda *a: None
    m = step(3)
    for kv in (first, second):
        r.kv = kv
        for l in range(2):
            r.attention_block(l, m)
            assert [t.data_ptr() for t in used] == [kv[l].data_ptr()] * 2
            used.clear()


def test_a_step_that_gets_other_sizes():
    r = HybridRunner.__new__(HybridRunner)
    r._columns, r._proj = [({"a": (0, 3), "b": (3, 2)}, 5, 0)], torch.zeros(100)
    m = step(6)
    first, parts = r._projection(0, m)
    assert first.shape == (6, 5) and r._projection(0, m)[0] is first and parts["b"].shape == (6, 2)
    m.num_tokens = 4
    assert r._projection(0, m)[0].shape == (4, 5)
    assert r._projection(0, dataclasses.replace(m, num_tokens=7))[1]["a"].shape == (7, 3)
