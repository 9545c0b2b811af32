"""Weight-streaming product at the edges of the eight tokens and the slices that its epilogue works in."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 3, 4, 5, 8, 9, 16, 17, 25, 61, 121, 128, 249])
@pytest.mark.parametrize("split", [1, 2, 3, 4, 8])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_token_groups(M, split, dtype):
    from blitz_scale_b200 import ops
    N, K = 328, 576                                  # three tiles, the last one partly filled; nine K blocks
    g = torch.Generator(device="cuda").manual_seed(M * 16 + split)
    r = lambda *s, dt=dtype: torch.randn(*s, generator=g, device="cuda").to(dt)
    a, b, gu, bias = r(M, K), r(K, N) * K ** -0.5, r(K, 2 * N) * K ** -0.5, r(2 * N)
    acc, ga = a.double() @ b.double(), a.double() @ gu.double()
    gate, up = ga[:, :N], ga[:, N:]
    # rounding of the output (2^-9 or 2^-12 of the value), sums of K products in fp32 (K 2^-24 of sums of size 1)
    rel = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11

    def check(out, ref, what, rel=rel):
        assert ((out[1:M + 1, 8:8 + N].double() - ref).abs() <= rel * ref.abs() + 1e-4).all(), what
        out[1:M + 1, 8:8 + N] = -7.0
        assert (out == -7.0).all(), f"{what}: written outside"

    def room(dt):
        out = torch.full((M + 2, N + 16), -7.0, device="cuda", dtype=dt)
        return out, out[1:M + 1, 8:8 + N]
    kw = dict(decode_path=True, decode_split=split, static_b=True)
    out, view = room(dtype)
    check((ops.gemm(a, b, out=view, **kw), out)[1], acc, "store")
    old = r(M, N)
    view.copy_(old)
    check((ops.gemm(a, b, out=view, residual=view, epilogue="add", **kw), out)[1], acc + old.double(), "add")
    check((ops.gemm(a, gu, out=view, epilogue="silu_mul", **kw), out)[1], gate * torch.sigmoid(gate) * up, "silu_mul")
    gb, ub = (gate + bias[:N].double()).clamp(max=3.0), (up + bias[N:].double()).clamp(-3.0, 3.0)
    check((ops.gemm(a, gu, out=view, epilogue="clamp_glu", bias=bias, alpha=3.0, beta=1.7, **kw), out)[1],
          gb * torch.sigmoid(1.7 * gb) * (ub + 1), "clamp_glu")
    out, view = room(torch.float32)
    check((ops.gemm(a, b, out=view, **kw), out)[1], acc, "store fp32", 1e-5)
    old = r(M, N, dt=torch.float32)
    view.copy_(old)
    check((ops.gemm(a, b, out=view, epilogue="axpy", alpha=0.8, **kw), out)[1], old.double() + 0.8 * acc, "axpy", 1e-5)
    check((ops.gemm(a, b, out=view, epilogue="softcap", alpha=2.0, **kw), out)[1], 2.0 * torch.tanh(acc / 2.0), "softcap", 1e-4)
    ops.check_status()
