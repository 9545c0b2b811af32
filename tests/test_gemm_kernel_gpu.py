"""Products without a hint, at the lines of the rule that names their kernel (tests/test_gemm_kernel_cpu.py), both sides."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("M,N,K,epi", [(300, 2048, 4096, "store"), (300, 2176, 4096, "add"), (300, 2048, 520, "add"), (300, 2048, 512, "axpy"),
                                       (3000, 128, 2048, "store"), (8448, 72, 576, "axpy"), (8449, 72, 576, "store")])
def test_default_dispatch(M, N, K, epi):
    from blitz_scale_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(M + K)
    a, w = torch.randn(M, K, device=DEV, generator=g).bfloat16(), (torch.randn(K, N, device=DEV, generator=g) * K ** -0.5).bfloat16()
    old = torch.randn(M, N, device=DEV, generator=g).to(torch.float32 if epi == "axpy" else torch.bfloat16)
    want = a.float() @ w.float() + (old.float() if epi != "store" else 0)
    out = ops.gemm(a, w, out=old.clone(), residual=old if epi == "add" else None, epilogue=epi)
    ops.check_status()
    number = {"store": 0, "add": 1, "axpy": 5}[epi]
    if ops.lib().blitz_gemm_kernel(M, N, K, number, 1) == 4:          # (the kernel that the rule names has run)
        same = ops.gemm(a, w, out=old.clone(), residual=old if epi == "add" else None, epilogue=epi, quad_path=True)
        assert torch.equal(out, same)
    # one rounding of the result, and 32-bit sums in another order
    assert float(((out.float() - want).abs() - (1e-5 if epi == "axpy" else 2.0 ** -8) * want.abs()).max()) <= 2e-5 * K ** 0.5
