"""Norms of wide rows on both sides of the number of blocks that the SMs hold at once."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H", [4096, 8192, 14336])
@pytest.mark.parametrize("more", [-1, 0, 1, 217])
def test_wide_rows(H, more):
    from blitz_scale_b200 import ops
    T = 2 * torch.cuda.get_device_properties(0).multi_processor_count + more
    g = torch.Generator(device="cuda").manual_seed(H + T)
    x, r, w = (torch.randn(*s, generator=g, device="cuda").bfloat16() for s in ((T, H), (T, H), (H,)))
    norm = lambda v: v * torch.rsqrt((v * v).mean(1, keepdim=True) + 1e-5) * w.double()
    want, both = norm(x.double()), (x.float() + r.float()).bfloat16()
    got = ops.rms_norm(x, w, 1e-5)
    # two roundings to 16 bits at most
    assert ((got.double() - want).abs() <= 2.0 ** -7 * want.abs() + 1e-6).all()
    got = ops.add_rms_norm(x, r, w, 1e-5)
    want = norm(both.double())
    assert torch.equal(r, both) and ((got.double() - want).abs() <= 2.0 ** -7 * want.abs() + 1e-6).all()
