"""RMS norm with a row's first columns kept in registers: widths below a warp, at and beyond what the threads keep, in place."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H", [8, 264, 8184, 8192, 8200, 16392])
@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
def test_rms_norm(H, dt):
    from blitz_scale_b200 import ops
    for T in (1, 149):
        x = torch.randn(T, H, device="cuda").to(dt)
        w = (1 + 0.1 * torch.randn(H, device="cuda")).to(dt)
        d = x.double()
        want = d * torch.rsqrt(d.pow(2).mean(-1, keepdim=True) + 1e-5) * w.double()
        out = torch.full((T + 1, H), 7.0, device="cuda", dtype=dt)
        ops.rms_norm(x, w, 1e-5, out=out[:T])
        # one rounding of the result (unit roundoff 2^-8 or 2^-11, subnormals 2^-25) and fp32 arithmetic
        assert bool(((out[:T].double() - want).abs() <= want.abs() * (2 ** -7.99 if dt == torch.bfloat16 else 2 ** -10.99) + 1e-7).all())
        assert bool((out[T] == 7.0).all())
        ops.rms_norm(x, w, 1e-5, out=x)
        assert torch.equal(x, out[:T])


@pytest.mark.parametrize("H", [8, 264, 4096, 4104, 8192, 8200, 16392])
@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
def test_add_rms_norm(H, dt):
    """With a residual, which is rounded before it is normed: rows below, at and beyond what the threads keep, more and fewer than SMs."""
    from blitz_scale_b200 import ops
    for T in (1, 149):
        x, r = torch.randn(T, H, device="cuda").to(dt), torch.randn(T, H, device="cuda").to(dt)
        w = (1 + 0.1 * torch.randn(H, device="cuda")).to(dt)
        total = x + r                                      # one rounding, as in the kernel
        d = total.double()
        want = d * torch.rsqrt(d.pow(2).mean(-1, keepdim=True) + 1e-5) * w.double()
        res, out = r.clone(), torch.full((T + 1, H), 7.0, device="cuda", dtype=dt)
        ops.add_rms_norm(x, res, w, 1e-5, out=out[:T])
        assert torch.equal(res, total)
        assert bool(((out[:T].double() - want).abs() <= want.abs() * (2 ** -7.99 if dt == torch.bfloat16 else 2 ** -10.99) + 1e-7).all())
        assert bool((out[T] == 7.0).all())
        res = r.clone()
        ops.add_rms_norm(x, res, w, 1e-5, out=x)           # over its input
        assert torch.equal(res, total) and torch.equal(x, out[:T])
