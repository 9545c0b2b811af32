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
    # (3, 5, 12, 18: parts or whole sequences as measured at 1000 tokens of 8 KV heads; 25 and 200 whole)
    for B, rows, want in [(1, 1, 8), (3, 4, 8), (5, 8, 4), (12, 16, 1), (18, 24, 1), (25, 32, 1), (200, 256, 1)]:
        batch = types.SimpleNamespace(size=B, max_seq_len=lambda: 1000, num_pages=lambda B=B: 16 * B, fill_decode=lambda *a: 0)
        with pytest.raises(Captured) as got:
            eng.decode(batch)
        assert got.value.args == (rows, want), (B, got.value.args)


# rows, KV heads, longest, tokens -> choice
RULE = [
    # contexts of a few chunks stay whole, whatever the batch
    *[((n, h, length, n * length), 1) for n in (1, 2, 3, 24, 100, 256) for h in (1, 2, 8) for length in (1, 64, 200, 300)],
    *[((n, 8, length, n * length // 2), 1) for n in (2, 16, 32, 61, 256) for length in (64, 300)],
    *[((n, 8, 600, n * 300), 1) for n in (16, 32, 61, 256)],
    # few heads and long contexts: as many parts as there are halves for
    ((1, 1, 100_000, 100_000), 32), ((1, 8, 100_000, 100_000), 32), ((2, 8, 16_000, 32_000), 16), ((1, 1, 1000, 1000), 8), ((1, 8, 1500, 1500), 8), ((1, 8, 1700, 1700), 16),
    ((1, 8, 500, 500), 8), ((1, 8, 4000, 4000), 16), ((5, 8, 4000, 20_000), 4),
    # second halves of SMs for parts of four and eight
    ((16, 4, 1000, 16_000), 4), ((16, 4, 3000, 48_000), 4), ((16, 4, 1000, 9000), 4), ((8, 4, 1000, 8000), 8), ((3, 8, 700, 2100), 8), ((9, 8, 1000, 9000), 1),
    # one length: whole where the SMs are full, ranges where a last round would be nearly empty
    ((256, 8, 513, 256 * 513), 1), ((37, 8, 4000, 37 * 4000), 1), ((38, 8, 4000, 38 * 4000), 0), ((64, 8, 4000, 64 * 4000), 1),
    ((38, 8, 200, 38 * 200), 1),
    # unequal: parts where there are few, else ranges
    ((2, 8, 600, 900), 8), ((2, 8, 4000, 4100), 8), ((5, 8, 1000, 3000), 4), ((16, 8, 16_000, 100_000), 0), ((61, 8, 3500, 61 * 1100), 0),
    ((200, 1, 16_000, 200 * 8000), 0),
    # more sequences than ranges are dealt out for
    ((257, 8, 4000, 257 * 1000), 1), ((300, 1, 1000, 300_000), 1),
]


@pytest.mark.parametrize("args,want", RULE)
def test_rule(args, want):
    assert E.decode_parts(*args) == want


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
    """Without them a batch of one length passes for an unequal one."""
    calls = [line for f in (ROOT / "bench.py", *(ROOT / "bench").glob("*.py")) for line in f.read_text().splitlines() if "choose_splits(" in line]
    assert calls and all("page_size" in line for line in calls)


# keys of the singles, keys of the portion, apart; 32 heads
SINGLES = [([60], 300, False), ([300], 300, False), ([1000], 1531, False), ([1000] * 3, 1531, False), ([300] * 2, 3842, False),
           ([1000] * 4, 3842, False), ([4000], 1531, True), ([1000] * 8, 1531, True), ([300] * 16, 1531, True), ([60] * 43, 300, True),
           ([1000] * 8, 3842, True), ([700] * 43, 3842, True)]


@pytest.mark.parametrize("singles,portion,apart", SINGLES)
def test_few_single_tokens_stay_beside_the_portion(singles, portion, apart):
    """What the step asks of its runner: leading rows that go through the decode kernels, out of those with one token."""
    eng = E.Engine.__new__(E.Engine)
    eng.cfg, eng.tp, eng.use_graphs, eng.max_batch = get_config("llama3_8b"), 1, False, 256
    eng.layout, eng.host_np, eng._h2d = types.SimpleNamespace(page_indices=0), None, lambda n: None
    n, kv = len(singles), [*singles, portion]

    class Asked(Exception):
        pass

    def views(T, rows, P, prefill, q_lens, splits, kv_lens, singles):
        raise Asked(singles)
    eng._views = views
    fill = lambda *a: (n + 100, 0, n + 1, n, list(range(n + 1)), [1] * n + [100], kv)
    with pytest.raises(Asked) as got:
        eng._step_pass(types.SimpleNamespace(fill_step=fill), [1] * n + [100], [])
    assert got.value.args == (n if apart else 0,)
