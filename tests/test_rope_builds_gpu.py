"""Rotation and cache write: as many tokens as four blocks an SM take at once and one more, which go to different builds of the kernel."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("interleaved", [False, True])
@pytest.mark.parametrize("qh,kvh,dim,rot", [(16, 4, 128, 64), (32, 8, 128, 128), (4, 2, 64, 32)])
@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16, torch.float32])
def test_both_builds(qh, kvh, dim, rot, interleaved, dt):
    from blitz_scale_b200 import ops
    threads = 128 if (qh + kvh) * dim <= 2048 else 256
    edge = 1024 // threads * torch.cuda.get_device_properties(0).multi_processor_count
    g = torch.Generator(device="cuda").manual_seed(dim + rot)
    freqs = ops.rope_freqs(rot, 1e5, "cuda")
    x = torch.randn(edge + 1, (qh + 2 * kvh) * dim, generator=g, device="cuda").to(dt)
    pos, slot = (torch.arange(edge + 1, device="cuda", dtype=torch.int32) * k for k in (37, 1))
    slot[5] = -1

    def run(pieces):
        y, kv = x.clone(), torch.zeros(edge // 64 + 1, 2, 64, kvh, dim, device="cuda", dtype=dt)
        a, b = qh * dim, (qh + kvh) * dim
        for lo, hi in pieces:
            p = y[lo:hi]
            ops.rope_store(p[:, :a], p[:, a:b], p[:, b:], pos[lo:hi], slot[lo:hi], kv, freqs, q_heads=qh, kv_heads=kvh, dim=dim, rot_dims=rot,
                           page_size=64, interleaved=interleaved)
        ops.check_status()
        return y.double(), kv.double()
    # x cos - y sin of the same angles, one rounding to the type and two in fp32 whichever way it is contracted; |x| + |y| stays below 12
    bound = 12 * {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11, torch.float32: 2.0 ** -23}[dt]
    for got, want in zip(run([(0, edge + 1)]), run([(0, edge), (edge, edge + 1)])):
        assert (got - want).abs().max() <= bound
