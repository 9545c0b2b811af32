"""The gated epilogue's quotient over the whole range of its argument, in every product kernel that has one."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw", [dict(decode_path=True, decode_split=1), dict(decode_path=True, decode_split=2), dict(wide_path=True),
                                dict(decode_path=False, pair_path=False, wide_path=False)], ids=["stream", "split", "wide", "tiles"])
def test_silu_over_its_range(kw):
    from blitz_scale_b200 import ops
    inf = float("inf")
    special = [0.0, -0.0, inf, float("nan"), 3e38, -3e38, 1e-38, -1e-38, 1e-40, -87.0, -87.5, -88.0, -89.0, -100.0, -104.0, 88.0, 1.0, -1.0]
    g = torch.Generator().manual_seed(5)
    x = torch.cat([torch.tensor(special), (torch.rand(4000, generator=g) - 0.5) * 180, torch.randn(2000, generator=g) * 3,
                   torch.logspace(-37, 2, 1000), -torch.logspace(-37, 2, 1000)]).to(torch.bfloat16)
    M, K, n = 64, 128, -(-x.numel() // 64)
    x = torch.cat([x, torch.zeros(M * n - x.numel(), dtype=torch.bfloat16)]).view(M, n)
    for c in range(0, n, K):          # column c + j of the gate is the j-th activation, the up columns are ones times the last activation, one
        part = x[:, c:c + K - 1]
        a = torch.zeros(M, K, dtype=torch.bfloat16)
        a[:, :part.shape[1]] = part
        a = torch.where(torch.isfinite(a), a, torch.zeros_like(a))
        a[:, K - 1] = 1.0
        eye = torch.zeros(K, 128, dtype=torch.bfloat16)
        eye[:K - 1, :K - 1] = torch.eye(K - 1, dtype=torch.bfloat16)
        up = torch.zeros(K, 128, dtype=torch.bfloat16)
        up[K - 1] = 1.0
        got = ops.gemm(a.cuda(), torch.cat([eye, up], 1).cuda(), epilogue="silu_mul", **kw).cpu().double()[:, :K - 1]
        z = a[:, :K - 1].double()
        want = z / (1 + torch.exp(-z))
        # e^-x to 2 units of fp32 beyond its argument's rounding (|x| 2^-24), one rounding to 16 bits, e^-x overflows fp32 from -88.7 on (results of 3e-37)
        bound = (2.0 ** -8 + 2.0 ** -22 * (1 + z.abs())) * want.abs() + 6e-37
        assert ((got - want).abs() <= bound).all(), (got - want).abs().max()
    # infinities and NaN behave as the plain formula in fp32
    a = torch.zeros(M, 64, dtype=torch.bfloat16)
    a[0, 0], a[1, 0], a[2, 0] = inf, -inf, float("nan")
    b = torch.zeros(64, 256, dtype=torch.bfloat16)
    b[0, :128] = 1.0
    b[1, 128:] = 1.0
    a[:, 1] = 1.0
    b2 = b.clone()
    got = ops.gemm(a.cuda(), b2.cuda(), epilogue="silu_mul", **kw).cpu()
    assert torch.isnan(got[1:3]).all() and (got[3:] == 0).all()
    ops.check_status()
