"""Decode attention over equal shares of all keys (num_splits = 0) against fp32 attention of every sequence by itself."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _reference(q, k, v, scale, kw, b, h, H):
    """Head h of sequence b: q [d], k [n, d], v [n, vd] in fp32."""
    n = k.shape[0]
    pos, j = n - 1, torch.arange(n, device=DEV)
    s = (k @ q) * scale
    if kw.get("softcap"):
        s = kw["softcap"] * torch.tanh(s / kw["softcap"])
    if kw.get("bias") is not None:
        table = kw["bias"][h].float()
        s = s + table[(pos - j).clamp(max=len(table) - 1)]
    see = torch.ones(n, dtype=torch.bool, device=DEV)
    w = kw.get("window", 0)
    if w:
        see = j // w == pos // w if kw.get("chunked") else (pos - j < w) | (j < kw.get("keep_first", 0))
    if kw.get("sigmoid"):
        p = torch.sigmoid(s) * see
    else:
        s = s.masked_fill(~see, float("-inf"))
        if kw.get("sink") is not None:
            s = torch.cat([s, kw["sink"][h].float().view(1)])
        p = torch.softmax(s, 0)[:n]
    o = p @ v
    return o * torch.sigmoid(kw["gate"][b, h].float()) if kw.get("gate") is not None else o


# sequences (0: a padding row), query and KV heads, key and value size, page
CASES = [
    ([978], 32, 8, 128, 128, 64, {}),                                  # fewer items than SMs: every CTA a chunk
    ([1], 8, 1, 64, 64, 16, {}),                                       # a single chunk in all
    ([0, 0, 5, 0], 8, 2, 64, 64, 64, {}),                              # rows of padding around it
    ([3, 700, 64, 65, 0, 2049, 1], 16, 4, 128, 128, 64, {}),
    ([513] * 150 + [40, 3000], 8, 8, 128, 128, 64, {}),                # whole items between two incomplete ones
    ([17, 900, 250, 2500], 12, 2, 128, 64, 64, {"gate": True}),        # values of another size
    ([600, 33, 1500], 12, 1, 64, 64, 32, {"sink": True, "window": 300, "keep_first": 70, "softcap": 20.0}),
    ([600, 33, 1500, 0], 8, 2, 128, 128, 64, {"window": 256, "chunked": True, "sigmoid": True, "bias": 1}),
    ([900, 130, 1], 8, 4, 64, 64, 64, {"bias": 40}),
    ([30 + 7 * i for i in range(256)], 4, 2, 64, 64, 64, {}),          # the largest batch
]


@pytest.mark.parametrize("case", range(len(CASES)))
@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
def test_shares_of_all_keys(case, dt):
    from blitz_scale_b200 import ops
    lens, H, G, d, dv, page, opts = CASES[case]
    g = torch.Generator(device=DEV).manual_seed(case)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g).to(dt)
    used = [-(-n // page) for n in lens]
    pages, B, scale = sum(used) + 3, len(lens), 1.3 * d ** -0.5
    perm = torch.randperm(pages, device=DEV, generator=g).to(torch.int32)
    pool = rnd(pages, 2, page, G, d) if dv == d else None
    kv = pool if dv == d else ops.KVPair(rnd(pages, page, G, d), rnd(pages, page, G, dv))
    keys, values = (pool[:, 0], pool[:, 1]) if dv == d else (kv.k, kv.v)
    starts = [sum(used[:i]) for i in range(B + 1)]
    indptr = torch.tensor(starts, dtype=torch.int32, device=DEV)
    last = torch.tensor([n - (u - 1) * page if n else 0 for n, u in zip(lens, used)], dtype=torch.int32, device=DEV)
    q = rnd(B, H * d + 8)[:, :H * d]
    kw = dict(opts)
    if "gate" in kw:
        kw["gate"] = rnd(B, H)
    if "sink" in kw:
        kw["sink"] = 2.0 + rnd(H)
    if "bias" in kw:
        kw["bias"] = rnd(H, kw["bias"])
    out = torch.full((B, H * dv), 7.0, dtype=dt, device=DEV)
    ops.attn_decode(q, kv, perm, indptr, last, q_heads=H, kv_heads=G, head_dim=d, page_size=page, num_splits=0, sm_scale=scale, out=out, **kw)
    ops.check_status()
    # probabilities and outputs are rounded to the type once each: at most its half unit, of values whose weights sum to one; sums of
    # weights that are not normalised grow with their number
    unit = 2.0 ** -8 if dt == torch.bfloat16 else 2.0 ** -11
    picks = range(B) if B < 20 else [0, 1, B // 2, B - 2, B - 1]
    for b in picks:
        n = lens[b]
        if n == 0:
            assert bool((out[b] == 0).all())
            continue
        rows = torch.arange(n, device=DEV)
        at = perm[starts[b]:starts[b + 1]].long()[rows // page]
        for h in range(H):
            k, v = keys[at, rows % page, h // (H // G)].float(), values[at, rows % page, h // (H // G)].float()
            want = _reference(q[b, h * d:(h + 1) * d].float(), k, v, scale, kw, b, h, H)
            got = out[b, h * dv:(h + 1) * dv].float()
            big = float(want.abs().max()) + float(v.abs().max()) * (0.1 if not kw.get("sigmoid") else 1.0)
            assert float((got - want).abs().max()) <= 3 * unit * big, (b, h)


def test_one_workspace_for_all_launches():
    """Launches of other batches, lengths and heads share a workspace, eagerly and in a graph: each leaves its tickets zero, and results
    repeat bit for bit.  The page tables are read before the kernel in front has finished."""
    from blitz_scale_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(5)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g).to(torch.bfloat16)
    calls, size = [], 0
    for lens, H, G, d, page in [([978], 32, 8, 128, 64), ([3, 700, 64, 65, 0, 2049, 1], 16, 4, 128, 64), ([900, 130, 1], 8, 4, 64, 64),
                                ([30 + 7 * i for i in range(256)], 4, 2, 64, 64), ([0, 0, 5, 0], 8, 2, 64, 16), ([600, 33, 1500], 12, 1, 64, 32)]:
        used = [-(-n // page) for n in lens]
        kv, q = rnd(sum(used) + 1, 2, page, G, d), rnd(len(lens), H * d)
        i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
        tables = (torch.randperm(sum(used) + 1, device=DEV, generator=g).to(torch.int32), i32([sum(used[:i]) for i in range(len(lens) + 1)]),
                  i32([n - (u - 1) * page if n else 0 for n, u in zip(lens, used)]))
        calls.append((q, kv, tables, dict(q_heads=H, kv_heads=G, head_dim=d, page_size=page, num_splits=0, static_table=True)))
        size = max(size, ops.attn_decode_workspace_bytes(len(lens), H, d, 0))
    want = [ops.attn_decode(q, kv, *t, **kw) for q, kv, t, kw in calls]              # (a fresh workspace each)
    ws = torch.zeros(size, dtype=torch.uint8, device=DEV)
    tickets = ws[:256 * 128 * 4]
    outs = [torch.full_like(w, 7.0) for w in want]
    norm_in, norm_w, norm_out = rnd(256, 4096), torch.ones(4096, dtype=torch.bfloat16, device=DEV), torch.empty(256, 4096, dtype=torch.bfloat16, device=DEV)

    def body():
        for (q, kv, t, kw), out in zip(calls, outs):
            ops.rms_norm(norm_in, norm_w, 1e-5, out=norm_out)                         # a kernel to run beside
            ops.attn_decode(q, kv, *t, workspace=ws, out=out, **kw)

    def same():
        ops.check_status()
        assert not bool(tickets.any())
        for out, w in zip(outs, want):
            assert torch.equal(out, w)
            out.fill_(7.0)
    for _ in range(2):
        body()
        same()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        body()
        body()
    for _ in range(3):
        graph.replay()
        same()
