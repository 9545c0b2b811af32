"""Linear attention over rows long enough to be cut into segments, against the recurrence token by token."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _err(a, b):
    a, b = a.float(), b.float()
    return (a - b).norm(dim=1) / b.norm(dim=1)


@pytest.mark.parametrize("form", ["gla", "wkv"])
@pytest.mark.parametrize("heads,dim,vdim,rank", [(2, 128, 128, 16), (1, 64, 64, 8), (3, 24, 72, 4), (16, 128, 256, 16)])
# ends of segments (256 tokens) and of chunks, with a short row between; second portions start from a state
@pytest.mark.parametrize("lens", [(2049,), (700, 3, 1536), (1024, 1025, 64)])
def test_rows_in_segments(form, heads, dim, vdim, rank, lens):
    from blitz_scale_b200 import ops
    if form == "wkv":
        vdim = dim
    gen = torch.Generator().manual_seed(dim + sum(lens))
    r = lambda *s: torch.randn(*s, generator=gen)
    bf = lambda t: t.to(DEV, torch.bfloat16)
    hk, hv, first = heads * dim, heads * vdim, 1          # a token of another row in front, as beside decoded tokens
    T = first + sum(lens)
    x = bf(torch.cat([r(T, hk), r(T, hk) * dim ** -0.5, r(T, hv), r(T, hv), r(T, (rank + 7) // 8 * 8)], 1))
    q, k, v, g, low = x.split([hk, hk, hv, hv, (rank + 7) // 8 * 8], 1)
    a2, a2_b = bf(r(rank, hk) * rank ** -0.5), bf(2.0 * r(hk) - (2.0 if form == "wkv" else 0.0))
    ends = [first + sum(lens[:i]) for i in range(len(lens) + 1)]
    i32 = lambda l: torch.tensor(l, dtype=torch.int32, device=DEV)
    slots, outs, states = i32([2 * i + 1 for i in range(len(lens))]), [], []
    for whole in (True, False):
        state = torch.full((2 * len(lens) + 1, heads, dim, vdim), 7.0, device=DEV)
        out = torch.zeros(2, T, hv, dtype=torch.bfloat16, device=DEV)
        for part in range(2):
            pos = i32([0] + [part * n + t for n in lens for t in range(n)])
            args = (pos, i32(ends), slots)
            if form == "gla":
                w, kw = (low, a2, a2_b, torch.ones(vdim, device=DEV, dtype=torch.bfloat16)), dict(rank=rank, tau=16.0, eps=1e-5)
                if whole:
                    ops.gla_recurrent(q, k, v, g, *w, state, out[part], *args, **kw)
                else:
                    ops.gla(q, k, v, g, *w, state, out[part], *args, row_lens=lens, **kw)
            else:
                w = (low.float().contiguous(), a2, a2_b, bf(torch.ones(hk)), torch.ones(hv, device=DEV, dtype=torch.bfloat16))
                # (a longest row below the chunked kernel's goes token by token)
                ops.wkv(q, k, v, g, *w, state, out[part], *args, rank=rank, eps=1e-5, row_lens=[1] if whole else lens)
        ops.check_status()
        outs.append(out[:, first:].reshape(-1, hv))
        states.append(state)
    # operands split into two bf16 numbers, outputs rounded to bf16 (2^-9 either side)
    err = _err(outs[1], outs[0])
    assert float(err.median()) < 6e-3 and int((err > 1.2e-2).sum()) <= len(err) // 25, (float(err.median()), float(err.max()))
    # no row is further off than two roundings to bf16 of every element (2^-8 each) and as much again by half for the arithmetic; the
    # first rows of every chunk, and so of every segment (4 chunks at least), which show a wrong starting state most, not even that
    assert float(err.max()) < 1.2e-2, float(err.max())
    starts = torch.zeros(2, sum(lens), dtype=torch.bool)
    for e, n in zip(ends, lens):
        starts[:, [e - first + t for t in range(n) if t % 64 < 8]] = True
    assert float(err[starts.reshape(-1).to(DEV)].max()) < 2 ** -7
    a, b = states[1][slots.long()], states[0][slots.long()]
    assert float((a - b).norm() / b.norm()) < 1e-4      # products of split operands: 2^-17 each
    assert bool((states[1][::2] == 7.0).all())


def test_rule_leaves_short_and_equal_rows_whole():
    from blitz_scale_b200 import ops
    scratch = ops.lib().blitz_gla_chunk_scratch
    assert scratch(200, 1, 200, 2, 128, 128) == 0 == scratch(64 * 40, 40, 64, 16, 128, 256) == scratch(300 * 8, 8, 300, 32, 128, 128)
    assert scratch(8192, 1, 8192, 1, 128, 128) > 0 and scratch(1 << 22, 65535, 1 << 20, 1, 8, 8) == 0
