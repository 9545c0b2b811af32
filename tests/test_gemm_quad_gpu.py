"""Products with K in two halves over a cluster of four, at the edges of rows, columns and K blocks, against sums in 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 96, 129, 200, 256, 257, 300, 512])
@pytest.mark.parametrize("N,K", [(64, 72), (72, 128), (136, 520), (256, 1088), (200, 1536), (4096, 576)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_halves_of_k(M, N, K, dtype):
    from blitz_scale_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(M * 16 + N)
    r = lambda *s, dt=dtype: torch.randn(*s, generator=g, device="cuda").to(dt)
    a, b = r(M, K), r(K, N) * K ** -0.5
    acc = a.double() @ b.double()
    # one rounding of a 16-bit output; sums of K products of size K^-0.5 in fp32
    rel = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11

    def check(out, ref, what, rel=rel):
        assert ((out[1:M + 1, 8:8 + N].double() - ref).abs() <= rel * ref.abs() + 1e-4).all(), what
        out[1:M + 1, 8:8 + N] = -7.0
        assert (out == -7.0).all(), f"{what}: written outside"

    def room(dt):
        out = torch.full((M + 2, N + 16), -7.0, device="cuda", dtype=dt)
        return out, out[1:M + 1, 8:8 + N]
    kw = dict(quad_path=True, static_b=True)
    out, view = room(dtype)
    check((ops.gemm(a, b, out=view, **kw), out)[1], acc, "store")
    old = r(M, N)
    view.copy_(old)
    check((ops.gemm(a, b, out=view, residual=view, epilogue="add", **kw), out)[1], acc + old.double(), "add")
    out, view = room(torch.float32)
    check((ops.gemm(a, b, out=view, **kw), out)[1], acc, "store fp32", 1e-5)
    old = r(M, N, dt=torch.float32)
    view.copy_(old)
    check((ops.gemm(a, b, out=view, epilogue="axpy", alpha=0.8, **kw), out)[1], old.double() + 0.8 * acc, "axpy", 1e-5)
    check((ops.gemm(a, b, out=view, epilogue="softcap", alpha=2.0, **kw), out)[1], 2.0 * torch.tanh(acc / 2.0), "softcap", 1e-4)
    assert torch.equal(ops.gemm(a, b, quad_path=True), ops.gemm(a, b, quad_path=True))
    ops.check_status()
