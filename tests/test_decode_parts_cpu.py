"""How a decode step divides its keys: the rule, and what the engine asks it (no GPU)."""
import pathlib
import types

import pytest

from blitz_scale_b200.models.config import get_config
from blitz_scale_b200.runtime import engine as E

ROOT = pathlib.Path(__file__).resolve().parents[1]


def test_rows_of_padding_do_not_count():
    """Sequences of one length are told from unequal ones by their own number, not by that of the graph's rows."""
    eng = E.Engine.__new__(E.Engine)
    eng.cfg, eng.tp, eng.use_graphs, eng.max_batch, eng.page_size, eng._graphs = get_config("llama3_8b"), 1, True, 256, 64, {}
    eng.status, eng.layout = types.SimpleNamespace(fully_loaded=lambda: True), types.SimpleNamespace(page_indices=0)
    eng.host_np, eng._h2d = None, lambda n: None

    class Captured(Exception):
        pass

    def capture(rows, splits):
        raise Captured(rows, splits)
    eng._capture = capture
    for B, rows, want in [(1, 1, 16), (3, 4, 8), (5, 8, 4), (12, 16, 2), (18, 24, 2), (200, 256, 1)]:
        batch = types.SimpleNamespace(size=B, max_seq_len=lambda: 1000, num_pages=lambda B=B: 16 * B, fill_decode=lambda *a: 0)
        with pytest.raises(Captured) as got:
            eng.decode(batch)
        assert got.value.args == (rows, want), (B, got.value.args)


def test_captures_cover_what_a_step_may_choose():
    """Every choice for one of the announced lengths is among the graphs of its bucket."""
    eng = E.Engine.__new__(E.Engine)
    eng.cfg, eng.tp, eng.use_graphs, eng.max_batch, eng._graphs = get_config("llama3_8b"), 1, True, 64, {}
    eng.pool, eng.host_np, eng.layout, eng._h2d = E.core.PagePool(4, 16), None, types.SimpleNamespace(page_indices=0), lambda n: None
    eng._capture = lambda rows, splits: eng._graphs.update({(rows, splits): None})
    saved = E.core.Batch, E.torch.cuda.current_stream
    E.core.Batch = lambda *a: types.SimpleNamespace(fill_decode=lambda *a: 0)
    E.torch.cuda.current_stream = lambda: types.SimpleNamespace(synchronize=lambda: None)
    try:
        assert eng.precapture(contexts=(64, 700, 1024)) == len(eng._graphs)
    finally:
        E.core.Batch, E.torch.cuda.current_stream = saved
    for n in range(1, 65):
        for length in (64, 700, 1024):
            for tokens in (n * length, length + n - 1):
                assert (E._bucket(n), eng.choose_splits(n, length, tokens)) in eng._graphs
    assert max(sum(rows == b for rows, _ in eng._graphs) for b in E._BUCKETS) <= 4


def test_every_caller_says_how_many_tokens():
    with pytest.raises(TypeError):
        E.Engine.choose_splits(E.Engine.__new__(E.Engine), 1, 1000)
    calls = [line for f in (ROOT / "bench.py", *(ROOT / "bench").glob("*.py")) for line in f.read_text().splitlines() if "choose_splits(" in line]
    assert calls and all("page_size" in line for line in calls)
