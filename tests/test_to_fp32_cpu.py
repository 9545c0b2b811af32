"""Copies in fp32 of tensors that live on the host, which no kernel may be given."""
import pytest
import torch

from blitz_scale_b200 import ops


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("shape", [(0, 8), (1, 8), (3, 40), (5, 33)])
def test_host_tensors(shape, dt, monkeypatch):
    monkeypatch.setattr(ops, "lib", lambda: pytest.fail("a kernel was asked for"))
    x = torch.randn(*shape).to(dt)
    got = ops.to_fp32(x)
    assert got.dtype == torch.float32 and torch.equal(got, x.float())
    assert got.data_ptr() != x.data_ptr() or not x.numel()
