"""Rotation and cache write with positions that are in place ahead of the projection, behind a projection that is still running."""
import pytest
import torch

pytestmark = pytest.mark.gpu
QH, KVH, HD, PAGE = 32, 8, 128, 16


def rotated(static, T, slot, a, w, pos, pages, dt):
    """The projection and the rotation, launched one behind the other with nothing between them."""
    from blitz_scale_b200 import ops
    qkv = torch.full((T, (QH + 2 * KVH) * HD), float("nan"), device="cuda", dtype=dt)    # what a rotation ahead of the projection would read
    kv = torch.zeros(pages, 2, PAGE, KVH, HD, device="cuda", dtype=dt)
    torch.cuda.synchronize()
    ops.gemm(a, w, out=qkv, static_b=True)
    ops.rope_kv_store(qkv, pos, slot, kv, q_heads=QH, kv_heads=KVH, head_dim=HD, page_size=PAGE, rope_theta=5e5, static_meta=static)
    return qkv, kv


@pytest.mark.parametrize("T", [1, 61, 300])
@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
def test_behind_a_projection(T, dt):
    from blitz_scale_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(T)
    # as deep as makes the projection (40 us and more) far longer than the angles take
    a, w = (torch.randn(*s, generator=g, device="cuda").to(dt) * s[1] ** -0.25 for s in ((T, 16384), (16384, (QH + 2 * KVH) * HD)))
    pos, slot = torch.arange(T, device="cuda", dtype=torch.int32) * 331, torch.arange(T, device="cuda", dtype=torch.int32)
    slot[T // 2] = -1
    want = rotated(False, T, slot, a, w, pos, T // PAGE + 1, dt)
    assert not torch.isnan(want[0]).any()
    for _ in range(5):
        got = rotated(True, T, slot, a, w, pos, T // PAGE + 1, dt)
        assert all(torch.equal(x, y) for x, y in zip(got, want))
    ops.check_status()


@pytest.mark.parametrize("static", [False, True])
def test_slot_beyond_the_cache(static):
    """The kernel's own bounds check reports it and leaves the cache alone; the rows are rotated all the same."""
    from blitz_scale_b200 import ops
    T, pages, dt = 5, 2, torch.bfloat16
    a, w = torch.randn(T, 256, device="cuda").to(dt), torch.randn(256, (QH + 2 * KVH) * HD, device="cuda").to(dt)
    pos = torch.arange(T, device="cuda", dtype=torch.int32) + 7
    good, slot = (torch.tensor(s, device="cuda", dtype=torch.int32) for s in ([0, 1, -1, 3, 4], [0, 1, pages * PAGE, 3, 4]))
    want = rotated(static, T, good, a, w, pos, pages, dt)
    ops.check_status()
    got = rotated(static, T, slot, a, w, pos, pages, dt)
    with pytest.raises(RuntimeError):
        ops.check_status()
    assert all(torch.equal(x, y) for x, y in zip(got, want))
    ops.check_status()          # (reading the status has cleared it)
