"""What is made at a device's first launch, asked for by two threads at once (no GPU)."""
import threading
import time

import pytest
import torch

from blitz_scale_b200 import ops


def _both(ask):
    start, got = threading.Barrier(2), [None, None]

    def run(i):
        start.wait()
        got[i] = ask()
    threads = [threading.Thread(target=run, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    return got


class _Lib:
    def __getattr__(self, name):
        return lambda *a: 64


@pytest.mark.parametrize("what", ["status_word", "gemm_workspace", "pair_gemm_workspace", "_status_ptr", "_scratch_of"])
def test_two_threads_get_the_same(monkeypatch, what):
    for table in ("_status", "_status_by_index", "_gemm_ws", "_pair_ws", "_gemm_scratch"):
        monkeypatch.setattr(ops, table, {})
    cpu, zeros = torch.device("cpu"), torch.zeros

    def slow(*a, **kw):
        time.sleep(0.05)
        return zeros(*a, **{**kw, "device": cpu})
    monkeypatch.setattr(torch, "zeros", slow)
    monkeypatch.setattr(torch, "empty", slow)
    monkeypatch.setattr(torch.cuda, "get_device_properties", lambda d: type("P", (), {"multi_processor_count": 148}))
    monkeypatch.setattr(ops, "lib", lambda: _Lib())
    word = zeros(1)
    ask = {"_status_ptr": lambda: ops._status_ptr(word), "_scratch_of": lambda: ops._scratch_of(0)}.get(what, lambda: getattr(ops, what)(cpu))
    a, b = _both(ask)
    assert a == b if isinstance(a, int) else a is b
    again = ask()
    assert again == a if isinstance(a, int) else again is a
