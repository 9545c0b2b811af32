"""Experts' rows added to an fp32 stream, and its norm: sizes at the edges of a thread's columns and of the rows in flight."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H", [8, 264, 2048, 4096, 4104, 8192, 8200])
@pytest.mark.parametrize("n", [1, 7, 8, 9, 17])
@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
def test_rows_in_flight(H, n, dt):
    from blitz_scale_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(H + n)
    T = 37
    x = torch.randn(T, H, generator=g, device="cuda")
    y, w = torch.randn(50, H, generator=g, device="cuda").to(dt), torch.randn(H, generator=g, device="cuda").to(dt)
    rows = torch.randint(0, 50, (T, n), generator=g, device="cuda")
    want = x.double() + y.double()[rows].sum(1)
    normed = want * torch.rsqrt((want * want).mean(1, keepdim=True) + 1e-3) * (1 + w.double())
    for keep_out in (True, False):
        xd, out = x.clone(), torch.empty(T, H, dtype=dt, device="cuda") if keep_out else None
        ops.stream_norm(xd, w if keep_out else None, 1e-3, out, w_offset=1.0, add=y, add_rows=rows.to(torch.int32))
        # sums of n + 1 numbers of size one in fp32; one rounding of the output
        assert ((xd.double() - want).abs() <= 2.0 ** -23 * (n + 1) * (1 + y.double().abs()[rows].sum(1))).all()
        if keep_out:
            assert ((out.double() - normed).abs() <= (2.0 ** -8 if dt == torch.bfloat16 else 2.0 ** -11) * normed.abs() + 1e-5).all()
    ops.check_status()


@pytest.mark.parametrize("H", [8, 264, 2048, 4096, 4104, 8192, 8200])
@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
def test_norm_alone(H, dt):
    from blitz_scale_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(H)
    x, w = torch.randn(37, H, generator=g, device="cuda"), torch.randn(H, generator=g, device="cuda").to(dt)
    before, out = x.clone(), torch.full((38, H), -7.0, device="cuda", dtype=dt)
    ops.stream_norm(x, w, 1e-3, out[:37], w_offset=1.0)
    want = x.double() * torch.rsqrt((x.double() ** 2).mean(1, keepdim=True) + 1e-3) * (1 + w.double())
    assert ((out[:37].double() - want).abs() <= (2.0 ** -8 if dt == torch.bfloat16 else 2.0 ** -11) * want.abs() + 1e-5).all()
    assert torch.equal(x, before) and (out[37] == -7.0).all()
    rows = torch.tensor([36, 0, 17], device="cuda", dtype=torch.int32)      # what the kernel for everything takes
    some = torch.empty(3, H, device="cuda", dtype=dt)
    ops.stream_norm(x, w, 1e-3, some, w_offset=1.0, rows=rows)
    assert ((some.double() - want[rows.long()]).abs() <= (2.0 ** -8 if dt == torch.bfloat16 else 2.0 ** -11) * want[rows.long()].abs() + 1e-5).all()
    ops.check_status()


@pytest.mark.parametrize("shape", [(1, 8), (3, 40), (7, 128256), (256, 32000), (5, 33)])
@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
def test_copy_in_32_bits(shape, dt):
    from blitz_scale_b200 import ops
    x = torch.randn(*shape, device="cuda").to(dt)
    x.view(-1)[:2] = torch.tensor([float("inf"), float("nan")], dtype=dt)
    assert torch.equal(ops.to_fp32(x).view(torch.int32), x.float().view(torch.int32))
    part = x[:, :shape[1] - 1]                      # not contiguous: the general copy
    got = ops.to_fp32(part)
    assert got.dtype == torch.float32 and torch.equal(got.view(torch.int32), part.float().view(torch.int32))


@pytest.mark.parametrize("T", [1, 61, 300])
def test_rotation_with_positions_known_ahead(T):
    from blitz_scale_b200 import ops
    outs = []
    for static in (False, True):
        g = torch.Generator(device="cuda").manual_seed(T)
        qkv = torch.randn(T, 12 * 64, generator=g, device="cuda").to(torch.bfloat16)
        pos, slot = torch.arange(T, device="cuda", dtype=torch.int32) * 331, torch.arange(T, device="cuda", dtype=torch.int32)
        slot[T // 2] = -1
        kv = torch.zeros(T // 16 + 1, 2, 16, 2, 64, device="cuda", dtype=torch.bfloat16)
        torch.cuda.synchronize()
        ops.rope_kv_store(qkv, pos, slot, kv, q_heads=8, kv_heads=2, head_dim=64, page_size=16, rope_theta=5e5, static_meta=static)
        outs.append((qkv, kv))
    assert all(torch.equal(a, b) for a, b in zip(*outs))
    ops.check_status()

