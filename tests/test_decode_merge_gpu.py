"""Decode attention in parts: both forms of the merge, at eight parts and beyond, at and beyond a warp's 32."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("splits", [2, 7, 8, 9, 32, 33, 40])
@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("with_sink", [False, True])
def test_parts(splits, hd, with_sink):
    from blitz_scale_b200 import ops
    B, qh, kvh, page, ctx = 3, 8, 2, 64, 2700
    g = torch.Generator(device="cuda").manual_seed(splits)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    npg = -(-ctx // page)
    kv, q, sink = rnd(B * npg, 2, page, kvh, hd), rnd(B, qh * hd), rnd(qh)
    idx, indptr = torch.arange(B * npg, device="cuda", dtype=torch.int32), torch.arange(B + 1, device="cuda", dtype=torch.int32) * npg
    last = torch.full((B,), ctx - (npg - 1) * page, device="cuda", dtype=torch.int32)
    ws = torch.zeros(max(1, ops.attn_decode_workspace_bytes(B, qh, hd, splits)), device="cuda", dtype=torch.uint8)
    got = ops.attn_decode(q, kv, idx, indptr, last, q_heads=qh, kv_heads=kvh, head_dim=hd, page_size=page, num_splits=splits, workspace=ws,
                          **(dict(sink=sink) if with_sink else {}))
    ops.check_status()
    k, v = (kv.double().view(B, npg, 2, page, kvh, hd)[:, :, i].reshape(B, npg * page, kvh, hd)[:, :ctx].repeat_interleave(qh // kvh, 2) for i in (0, 1))
    z = torch.einsum("bhd,bnhd->bhn", q.double().view(B, qh, hd), k) * hd ** -0.5
    z = torch.cat([z, sink.double()[None, :, None].expand(B, qh, 1)], 2) if with_sink else z
    w = torch.softmax(z, 2)[:, :, :ctx]
    want, room = (torch.einsum("bhn,bnhd->bhd", w, x) for x in (v, v.abs()))
    # probabilities and the result rounded to 16 bits once each, scores and sums in fp32
    assert ((got.double().view(B, qh, hd) - want).abs() <= 2.0 ** -8 * (want.abs() + 1.1 * room) + 1e-4).all()
