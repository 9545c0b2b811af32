"""The gated epilogue of every product kernel at the limits of its argument: subnormal reciprocals, sums that overflow, NaN."""
import pytest
import torch

from test_silu_gpu import test_silu_over_its_range as over_its_range

pytestmark = pytest.mark.gpu


def test_range_on_pairs():
    over_its_range(dict(pair_path=True))


@pytest.mark.parametrize("kw", [dict(decode_path=True, decode_split=1), dict(decode_path=True, decode_split=2), dict(wide_path=True),
                                dict(pair_path=True), dict(decode_path=False, pair_path=False, wide_path=False)],
                         ids=["stream", "split", "wide", "pairs", "tiles"])
def test_limits(kw):
    from blitz_scale_b200 import ops
    M, inf = 64, float("inf")
    # denominators beyond 2^126, whose reciprocal is subnormal: up values that bring the quotient back among the normal numbers
    z = torch.arange(-88.5, -80.0, 0.5, dtype=torch.float64)
    a = torch.zeros(M, 64, dtype=torch.bfloat16)
    a[:z.numel(), 0], a[:, 1] = z.to(torch.bfloat16), 1.0
    b = torch.zeros(64, 256, dtype=torch.bfloat16)
    b[0, :128], b[1, 128:] = 1.0, 2.0 ** 100
    got = ops.gemm(a.cuda(), b.cuda(), epilogue="silu_mul", **kw).cpu().double()[:z.numel()]
    want = (z / (1 + torch.exp(-z)) * 2.0 ** 100)[:, None]
    assert ((got - want).abs() <= (2.0 ** -8 + 2.0 ** -22 * (1 + z.abs()))[:, None] * want.abs()).all()
    # sums that overflow fp32, beside up values of one: x / (1 + e^-x) of an infinity is itself, of a negative one NaN
    a = torch.zeros(M, 64, dtype=torch.bfloat16)
    a[0, 0], a[1, 0], a[:, 1] = 3e38, -3e38, 1.0
    b[0, :128], b[1, 128:] = 4.0, 1.0
    got = ops.gemm(a.cuda(), b.cuda(), epilogue="silu_mul", **kw).cpu()
    assert (got[0] == inf).all() and torch.isnan(got[1]).all() and (got[2:] == 0).all()
    # a NaN stays one
    a[0, 0] = float("nan")
    got = ops.gemm(a.cuda(), b.cuda(), epilogue="silu_mul", **kw).cpu()
    assert torch.isnan(got[:2]).all() and (got[2:] == 0).all()
    ops.check_status()
