"""Decode graphs after a ragged step that asked for a larger scratch: they write into the buffer they were captured with."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _run(graphs: bool, monkeypatch):
    from blitz_scale_b200 import ops
    from blitz_scale_b200.runtime import core, engine
    from blitz_scale_b200.runtime.engine import Engine
    torch.cuda.set_device(0)
    monkeypatch.setattr(engine, "singles_apart", lambda *a: True, raising=False)
    eng = Engine("tiny_gpu", num_pages=128, page_size=16, max_batch=16, max_batch_tokens=512, seed=0, use_graphs=graphs)
    eng.choose_splits = lambda B, *a, **kw: 4            # scratch in proportion to the rows
    one = eng.new_batch(0, [core.SeqSpec(0, list(range(5, 305)), 4)])
    many = eng.new_batch(1, [core.SeqSpec(i, list(range(7 + i, 107 + i)), 4) for i in range(1, 11)])
    eng.step(one, [250])
    out = [eng.step(one, [1], [[0]])]                    # (captures the graph of one row)
    eng.step(many, [50] * 10)
    out.append(eng.step(many, [1] * 9 + [30], [[0]] * 9 + [[29]]))
    size = ops.attn_decode_workspace_bytes(1, eng.cfg.q_heads, eng.cfg.head_dim, 4)
    blocks = [torch.full((size,), 0x5A, dtype=torch.uint8, device="cuda") for _ in range(64)]
    out += [eng.step(one, [1], [[0]]) for _ in range(3)]
    ops.check_status()
    assert all(bool((b == 0x5A).all()) for b in blocks)
    return out


def test_graph_after_a_larger_scratch(monkeypatch):
    for a, b in zip(_run(True, monkeypatch), _run(False, monkeypatch)):            # the same kernels with the same parts
        assert torch.equal(a, b)
