"""Serving work of this framework on one GPU, through the engine that its workers and its trace replay call.

A case is one pass of a model that an engine holds: prompts (`Engine.prefill`), one token of every sequence (`Engine.step`,
which replays the decode graph), or a step that carries portions of prompts beside single tokens (`Engine.step`, ragged).

Models: the headline benchmark's shape (`llama3_8b`, 32 layers) and the designs whose layers differ at the sizes of their
benchmarks (8 layers).  Weights are random, of the scales that trained models have: every sublayer adds a part of the
stream's size, scores and router logits are of order one.

A state is a set of requests on an engine.  The engine (weights, graphs, workspaces) is what a serving process keeps for
all its requests, so it is made once per model; prompts, cached keys and values and recurrent states are the state's own.

Outputs are logits of the rows that a serving step wants (tokens are their arg-max, which near-ties would decide at
random here) and, after prompts, the whole cache that the pass has filled.  A decode step is repeated at its place: its
keys and values land where they were, and are read by the attention of the same step.
"""
import gc
import math
import random

import torch

PAGE = 64                       # tokens of a cache page
MAX_BATCH, MAX_TOKENS = 256, 8192
DTYPES = {"bfloat16": torch.bfloat16, "float16": torch.float16}

# ---------------------------------------------------------------------------------------------------------- models
LLAMA = dict(vocab=128256, hidden=4096, layers=32, heads=32, kv_heads=8, dim=128, inter=14336, theta=5e5, eps=1e-5)
VOCAB, LAYERS = 32000, 8


def _fafudra(H, ff, heads, kv, gla_heads, width, blocks):
    kinds = {"attention": dict(heads=heads, kv_heads=kv, dim=128, vdim=128, mask=dict(size=2048, keep_first=4),
                               rot=dict(base=1e5, dims=128), scale=128 ** -0.5, softcap=50.0),
             "gla": dict(heads=gla_heads, dim=128, vdim=256, tau=16.0, rank=16), "rglru": dict(width=width, blocks=blocks, conv=4)}
    return dict(architecture="Fafudra", norm=dict(eps=1e-6), residual_mult=0.8, vocab=VOCAB, width=H,
                layers=[dict(type=t, mixer=kinds[t], mlp=dict(ff=ff, kind="dense")) for t in ("gla", "attention", "rglru", "gla") * (LAYERS // 4)])


def _komulorn(H, heads, kv, vdim, E, top, ff, shared):
    rot = dict(base=5e5, dims=64, scaling=dict(factor=4.0, original=4096.0, fast=32.0, slow=1.0))
    mixer = dict(heads=heads, kv_heads=kv, dim=128, vdim=vdim, rot=rot, scale=128 ** -0.5)
    mlp = dict(kind="moe", router=dict(experts=E, top=top), expert=dict(ff=ff), shared=dict(ff=shared))
    return dict(architecture="Komulorn", norm=dict(eps=1e-6), vocab=VOCAB, width=H, logit_softcap=30.0,
                layers=[dict(type="attention", mixer=dict(mixer, **({"kv_from": i - 1} if i % 2 else {})), mlp=mlp) for i in range(LAYERS)])


def _vofidra(H, heads, kv, latent, E, identity, top, groups, keep, ff, dense):
    a = dict(heads=heads, kv_heads=kv, dim=128, vdim=128, scale=128 ** -0.5, bias_max=512, q_temp=dict(coef=0.1, every=2048), rows=32)
    b = dict(latent, scale=(latent["dim"] + latent["rot_dim"]) ** -0.5, rot=dict(base=5e5, dims=latent["rot_dim"]))
    moe = dict(kind="moe", router=dict(experts=E, identity=identity, top=top, groups=dict(count=groups, keep=keep)), expert=dict(ff=ff))
    return dict(architecture="Vofidra", norm=dict(eps=1e-6), vocab=VOCAB, width=H, logit_softcap=30.0, streams=4,
                layers=[dict(type="latent_attention" if i % 2 else "attention", mixer=b if i % 2 else a, mlp=moe if i else dict(kind="dense", ff=dense))
                        for i in range(LAYERS)])


def _norusun(H, ff, heads, kv, wkv, latent, ssd):
    wk = dict(heads=wkv[0], dim=wkv[1], rank=wkv[2])
    la = dict(latent, scale=(latent["dim"] + latent["rot_dim"]) ** -0.5, rot=dict(base=5e5, dims=latent["rot_dim"]), mask=dict(size=2048))
    left = dict(heads=heads, kv_heads=kv, dim=128, vdim=128, scale=128 ** -0.5, rot=dict(base=5e5, dims=128), mask=dict(size=2048))
    kinds = {"wkv": wk, "latent_attention": la, "parallel": dict(left=left, right=dict(ssd, conv=4))}
    return dict(architecture="Norusun", canon=dict(taps=4), norm=dict(eps=1e-5), vocab=VOCAB, width=H, streams=2,
                layers=[dict(type=t, mixer=kinds[t], mlp=None if t == "wkv" else dict(kind="dense", ff=ff, limit=7.0))
                        for t in ("wkv", "latent_attention", "parallel", "latent_attention") * (LAYERS // 4)])


HYBRID = {
    "fafudra_h4096": _fafudra(4096, 14336, 32, 8, 16, 4096, 16),
    "fafudra_h2048": _fafudra(2048, 8192, 16, 4, 8, 2048, 8),
    "komulorn_h2048": _komulorn(2048, 16, 4, 64, 64, 6, 1408, 2816),
    "vofidra_h2048": _vofidra(2048, 16, 4, dict(heads=32, dim=64, rot_dim=32, vdim=64, q_rank=768, kv_rank=256), 64, 16, 8, 8, 4, 1408, 8192),
    "norusun_h4096": _norusun(4096, 14336, 32, 8, (32, 128, 64), dict(heads=32, dim=96, rot_dim=32, vdim=128, q_rank=1024, kv_rank=512),
                              dict(heads=64, vdim=64, state=128, groups=8, norm_groups=8)),
    "norusun_h2048": _norusun(2048, 8192, 16, 4, (16, 128, 64), dict(heads=32, dim=64, rot_dim=32, vdim=64, q_rank=768, kv_rank=256),
                              dict(heads=32, vdim=64, state=128, groups=4, norm_groups=4)),
}


# ---------------------------------------------------------------------------------------------------------- cases
def _case(name, model, what, sequences, tokens, ragged=False, chunk=0, prefix=0, dtype="bfloat16"):
    """`sequences` prompts of `tokens` tokens in all, or contexts of single tokens; `chunk` tokens of one more prompt, `prefix` of
    which are cached already."""
    return {"name": name, "model": model, "pass": what, "sequences": sequences, "tokens": tokens, "ragged": ragged, "chunk": chunk,
            "prefix": prefix, "dtype": dtype}


def listed():
    return [
        # one user's request, token by token: latency, launches and the weight stream
        _case("llama decode 1", "llama3_8b", "decode", 1, 977),
        # the headline benchmark: a full decode batch
        _case("llama decode 256", "llama3_8b", "decode", 256, 256 * 512),
        # what continuous batching makes of traffic: requests of very different ages, the second 16-bit type
        _case("llama decode 61 ragged", "llama3_8b", "decode", 61, 61 * 1100, ragged=True, dtype="float16"),
        # time to the first token of one short prompt
        _case("llama prefill 117", "llama3_8b", "prefill", 1, 117),
        # a full prefill batch of prompts of unequal lengths
        _case("llama prefill 8192 ragged", "llama3_8b", "prefill", 9, 8192, ragged=True),
        # chunked prefill beside decode: a portion of a long prompt and the tokens of a running batch
        _case("llama step 1531 + 43", "llama3_8b", "step", 43, 43 * 700, ragged=True, chunk=1531, prefix=2311),
        # the designs whose layers differ: prompts and decode of windowed attention beside gated linear attention and recurrence
        _case("fafudra prefill 4999 ragged", "fafudra_h4096", "prefill", 4, 4999, ragged=True),
        _case("fafudra decode 48", "fafudra_h2048", "decode", 48, 48 * 700, ragged=True),
        # ... of a mixture of experts with shared caches
        _case("komulorn prefill 4096", "komulorn_h2048", "prefill", 8, 4096),
        _case("komulorn decode 16", "komulorn_h2048", "decode", 16, 16 * 1000),
        # ... of latent attention and experts over several streams, portions of prompts beside decode
        _case("vofidra step 773 + 24", "vofidra_h2048", "step", 24, 24 * 500, ragged=True, chunk=773, prefix=600),
        # ... of linear attention, latent attention in a window and a state space
        _case("norusun prefill 3001 ragged", "norusun_h4096", "prefill", 3, 3001, ragged=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    model = rng.choice(["llama3_8b"] * 6 + sorted(HYBRID))
    what = rng.choice(["decode", "decode", "prefill", "prefill", "step"])
    dtype = rng.choice(["bfloat16", "bfloat16", "float16"]) if model == "llama3_8b" else "bfloat16"
    most = 131072 if model == "llama3_8b" else 49152        # tokens of context in all
    if what == "prefill":
        tokens = _log(rng, 24, MAX_TOKENS)
        case = _case("", model, what, min(tokens, _log(rng, 1, 32)), tokens, rng.random() < 0.7, dtype=dtype)
    else:
        n = _log(rng, 1, MAX_BATCH if what == "decode" else 128)
        case = _case("", model, what, n, n * _log(rng, 60, min(4000, most // n)), rng.random() < 0.7, dtype=dtype)
        if what == "step":
            case.update(chunk=_log(rng, 32, 4096), prefix=rng.choice([0, _log(rng, 16, 4000)]))
    del case["name"]
    return case


def _lengths(case):
    """Tokens of every prompt, or of every context: equal, or spread over a factor of sixteen.  A matter of the case alone."""
    n, total = case["sequences"], case["tokens"]
    rng = random.Random(n * 1000003 + total)
    w = [math.exp(rng.uniform(0.0, math.log(16.0))) if case["ragged"] else 1.0 for _ in range(n)]
    out = [max(1, int(total * x / sum(w))) for x in w]
    while sum(out) != total:
        i = rng.randrange(n)
        out[i] += 1 if sum(out) < total else -1 if out[i] > 1 else 0
    return out


def _requests(case):
    """(tokens cached before the pass, tokens of the pass) of every request."""
    if case["pass"] == "prefill":
        return [(0, n) for n in _lengths(case)]
    return [(n, 1) for n in _lengths(case)] + ([(case["prefix"], case["chunk"])] if case["pass"] == "step" else [])


def _vocab(model):
    return LLAMA["vocab"] if model == "llama3_8b" else HYBRID[model]["vocab"]


def _prompts(case, seed):
    g = torch.Generator().manual_seed(seed * 7919 + 17)
    return [torch.randint(0, _vocab(case["model"]), (a + b,), generator=g).tolist() for a, b in _requests(case)]


# ---------------------------------------------------------------------------------------------------------- weights
def _normal(gen, shape, scale, mean=0.0, dtype=torch.bfloat16):
    t = torch.empty(shape, device="cuda", dtype=dtype).normal_(mean, 1.0, generator=gen)
    return t if scale == 1.0 and mean == 0.0 else ((t - mean) * scale + mean)


def _llama_shapes():
    c = LLAMA
    H, q, kv, ff = c["hidden"], c["heads"] * c["dim"], c["kv_heads"] * c["dim"], c["inter"]
    out = [("embed", (c["vocab"], H))]
    for l in range(c["layers"]):
        out += [(f"layers.{l}.{n}", s) for n, s in (("input_ln", (H,)), ("qkv", (H, q + 2 * kv)), ("o", (q, H)), ("post_ln", (H,)),
                                                    ("gate_up", (H, 2 * ff)), ("down", (ff, H)))]
    return out + [("final_norm", (H,)), ("lm_head", (H, c["vocab"]))]


def _llama_weight(i, name, shape, dtype):
    """Matrices [in, out]; a sublayer adds about a quarter of the stream's size."""
    gen = torch.Generator(device="cuda").manual_seed(1000 + i)
    kind = name.split(".")[-1]
    if len(shape) == 1:
        return _normal(gen, shape, 0.1, 1.0, dtype)
    scale = {"embed": 1.0, "qkv": 1.3, "o": 0.6, "gate_up": 1.0, "down": 0.5, "lm_head": 3.0}[kind]
    return _normal(gen, shape, scale if kind == "embed" else scale * shape[0] ** -0.5, dtype=dtype)


def _hybrid_weights(c):
    """Checkpoint tensors of a design's configuration (linear weights [out, in])."""
    gen, w = torch.Generator(device="cuda").manual_seed(4242), {}
    r = lambda *s, scale=1.0, mean=0.0: _normal(gen, s, scale, mean)
    lin = lambda o, i, scale=1.0: r(o, i, scale=scale * i ** -0.5)
    H, S, kind = c["width"], c.get("streams", 0), c["architecture"]

    def gains(name):
        if kind == "Vofidra":
            w[name], w[name + ".b"], w[name + ".alpha"] = r(H, scale=0.2, mean=1.2), r(H, scale=0.1), r(1, scale=0.05, mean=0.6).view(())
        elif kind == "Norusun":
            w[name] = r(1, scale=0.1, mean=1.2).view(())
        else:
            w[name] = r(H, scale=0.2, mean=0.0 if kind == "Fafudra" else 1.0)

    def attention(p, m):
        for n, heads, d in (("q", m["heads"], m["dim"]), ("k", m["kv_heads"], m["dim"]), ("v", m["kv_heads"], m["vdim"])):
            if (n == "v" and kind == "Fafudra") or (n != "q" and "kv_from" in m):
                continue
            w[p + n] = lin(heads * d, H, 1.3 if n != "v" else 1.0)
            if kind == "Komulorn":
                w[f"{p}{n}.b"] = r(heads * d, scale=0.3)
        w[p + "o"] = lin(H, m["heads"] * m["vdim"], 0.6)

    w["embed"] = r(c["vocab"], H, scale=0.5 if kind == "Fafudra" else 1.0)
    gains("final.norm")
    if kind == "Fafudra":
        w["final.norm"] = r(H, mean=-1.0)
    else:
        w["head"] = lin(c["vocab"], H, 3.0)
    for i, L in enumerate(c["layers"]):
        p, q, m, f = f"l{i}.mix.", f"l{i}.mlp.", L["mixer"], L["mlp"]
        for k in (1, 2) if f and kind != "Fafudra" else (1,):
            gains(f"l{i}.norm{k}")
            if S:
                w[f"l{i}.hc{k}.in"], w[f"l{i}.hc{k}.out"] = r(S, scale=0.2 / S, mean=1.0 / S), r(S, scale=0.2, mean=0.8)
                w[f"l{i}.hc{k}.mix"] = 0.9 * torch.eye(S, device="cuda", dtype=torch.bfloat16) + r(S, S, scale=0.05)
        if kind == "Norusun":
            w[f"l{i}.canon1"] = r(H, c["canon"]["taps"], scale=0.2)
        if L["type"] == "attention":
            attention(p, m)
            if kind == "Fafudra":
                w[p + "sink"] = r(m["heads"], mean=2.0)
            elif kind == "Komulorn":
                w[p + "g"] = lin(m["heads"], H)
            else:
                w[p + "q.norm"], w[p + "k.norm"] = r(m["dim"], scale=0.2, mean=1.2), r(m["dim"], scale=0.2, mean=1.2)
                w[p + "rel"] = r(m["rows"], m["heads"])
        elif L["type"] == "latent_attention":
            h, d, rd = m["heads"], m["dim"], m["rot_dim"]
            w[p + "dq"], w[p + "dkv"] = lin(m["q_rank"], H), lin(m["kv_rank"] + rd, H)
            w[p + "dq.norm"], w[p + "dkv.norm"] = r(m["q_rank"], scale=0.2, mean=1.0), r(m["kv_rank"], scale=0.2, mean=1.0)
            w[p + "uq"], w[p + "uk"], w[p + "uv"] = lin(h * (d + rd), m["q_rank"], 1.3), lin(h * d, m["kv_rank"], 1.3), lin(h * m["vdim"], m["kv_rank"])
            if kind == "Vofidra":
                w[p + "g"] = lin(h, H)
            else:
                w[p + "sink"] = r(h, mean=2.0)
            w[p + "o"] = lin(H, h * m["vdim"], 0.6)
        elif L["type"] == "gla":
            hk, hv = m["heads"] * m["dim"], m["heads"] * m["vdim"]
            for n, o in (("q", hk), ("k", hk), ("v", hv), ("g", hv), ("a1", m["rank"])):
                w[p + n] = lin(o, H)
            w[p + "a2"], w[p + "a2.b"], w[p + "norm"] = lin(hk, m["rank"], 2.0), r(hk, scale=2.0, mean=1.0), r(m["vdim"], scale=0.2, mean=1.0)
            w[p + "o"] = lin(H, hv, 0.6)
        elif L["type"] == "rglru":
            W, b = m["width"], m["width"] // m["blocks"]
            for n in ("y", "x"):
                w[p + n], w[f"{p}{n}.b"] = lin(W, H), r(W, scale=0.3)
            w[p + "conv"], w[p + "conv.b"] = r(W, m["conv"], scale=0.6), r(W, scale=0.3)
            for n in ("ra", "ri"):
                w[p + n], w[f"{p}{n}.b"] = r(m["blocks"], b, b, scale=b ** -0.5), r(m["blocks"], b, scale=0.5)
            w[p + "lam"], w[p + "o"] = r(W, scale=1.5, mean=-3.0), lin(H, W, 0.6)
        elif L["type"] == "wkv":
            n = m["heads"] * m["dim"]
            for s in "rkvgw":
                w[f"{p}mu.{s}"] = r(H, scale=0.25, mean=0.5)
            for s in "rkvg":
                w[p + s] = lin(n, H)
            w[p + "w1"], w[p + "w2"], w[p + "w0"] = lin(m["rank"], H), lin(n, m["rank"]), r(n, scale=0.8, mean=-1.5)
            w[p + "u"], w[p + "norm"], w[p + "o"] = r(m["heads"], m["dim"], scale=0.5, mean=0.5), r(n, scale=0.2, mean=1.0), lin(H, n, 0.6)
        else:
            a, b = m["left"], m["right"]
            attention(p + "left.", a)
            w[p + "left.q.norm"], w[p + "left.k.norm"] = r(a["heads"] * a["dim"], scale=0.2, mean=1.2), r(a["kv_heads"] * a["dim"], scale=0.2, mean=1.2)
            w[p + "left.pb"] = r(a["heads"], mean=-3.0)
            n, ch = b["heads"] * b["vdim"], b["heads"] * b["vdim"] + 2 * b["groups"] * b["state"]
            w[p + "right.in"], w[p + "right.o"] = lin(n + ch + b["heads"], H), lin(H, n, 0.6)
            w[p + "right.conv"], w[p + "right.conv.b"] = r(ch, b["conv"], scale=0.5), r(ch, scale=0.2)
            w[p + "right.dt_bias"], w[p + "right.A_log"], w[p + "right.D"] = r(b["heads"], scale=0.7, mean=-2.0), r(b["heads"], scale=0.7, mean=-0.5), r(b["heads"], scale=0.5, mean=1.0)
            w[p + "right.norm"] = r(n, scale=0.2, mean=1.0)
            w[p + "left.out"], w[p + "right.out"] = r(H, scale=0.1, mean=0.4), r(H, scale=0.1, mean=0.4)
        if f and f["kind"] == "dense":
            ff = f["ff"]
            w[q + "gate"], w[q + "up"], w[q + "down"] = lin(ff, H), lin(ff, H), lin(H, ff, 0.5)
            if kind == "Norusun":
                w[q + "gate.b"], w[q + "up.b"], w[q + "down.b"] = r(ff, scale=0.3), r(ff, scale=0.3), r(H, scale=0.1)
        elif f:
            # a layer's experts add little to the stream, so that the choices that rounding decides (a token's router scores
            # are often near one another) change the logits by no more than rounding does
            n, ff = f["router"]["experts"], f["expert"]["ff"]
            w[q + "router"] = lin(n + f["router"].get("identity", 0), H, 2.0)
            if kind == "Vofidra":
                w[q + "correction"] = r(n + f["router"]["identity"], scale=0.02)
            for e in range(n):
                if kind == "Vofidra":
                    w[f"{q}e{e}.gate"] = lin(ff, H)
                w[f"{q}e{e}.up"], w[f"{q}e{e}.down"] = lin(ff, H), lin(H, ff, 0.1 if kind == "Vofidra" else 0.03)
            if f.get("shared"):
                n = f["shared"]["ff"]
                w[q + "shared.up"], w[q + "shared.down"], w[q + "shared.sg"] = lin(n, H), lin(H, n, 0.3), lin(1, H)
    return w


# ---------------------------------------------------------------------------------------------------------- engine and states
_held = {}                      # the engine in use, by model and type


class _Reader:
    """Checkpoint tensors by name."""

    def __init__(self, tensors):
        self.tensors = tensors

    def get(self, name):
        return self.tensors[name]


def _engine(model, dtype):
    key = (model, dtype)
    if key not in _held:
        _held.clear()
        gc.collect()
        torch.cuda.empty_cache()
        from blitz_scale_b200.models.config import design_module, get_config
        from blitz_scale_b200.runtime.engine import Engine
        more = dict(page_size=PAGE, max_batch=MAX_BATCH, max_batch_tokens=MAX_TOKENS, dtype=DTYPES[dtype], ready=False)
        if model == "llama3_8b":
            eng = Engine(get_config(model), num_pages=3 * (131072 // PAGE + 320), **more)
            for i, (name, shape) in enumerate(_llama_shapes()):
                eng.seg[name].copy_(_llama_weight(i, name, shape, DTYPES[dtype]))
        else:
            w = _hybrid_weights(HYBRID[model])
            design = design_module(HYBRID[model]["architecture"].lower())
            cfg = design.parse_config(HYBRID[model], {n: tuple(t.shape) for n, t in w.items()}, name=model)
            eng = Engine(cfg, num_pages=3 * (49152 // PAGE + 400), state_slots=3 * MAX_BATCH + 32, **more)
            eng.seg.buffer.copy_(design.to_segment(_Reader(w), cfg, DTYPES[dtype]).buffer)
        eng.set_status_ready()
        _held[key] = eng
    return _held[key]


def _cached_llama(case, seed, layer, pages):
    """Keys and values of a layer's pages: of size one, as rotation leaves keys."""
    gen = torch.Generator(device="cuda").manual_seed(seed * 131 + layer)
    return torch.empty(pages, 2, PAGE, LLAMA["kv_heads"], LLAMA["dim"], device="cuda", dtype=DTYPES[case["dtype"]]).normal_(generator=gen)


def prepare(case, seed):
    from blitz_scale_b200.runtime import core
    eng = _engine(case["model"], case["dtype"])
    reqs, prompts = _requests(case), _prompts(case, seed)
    specs = [core.SeqSpec(i, p, 8) for i, p in enumerate(prompts)]
    state = {"engine": eng, "case": case}
    if case["pass"] == "prefill":
        # a pool of these prompts' pages, so that the pass fills the same part of the cache each time
        pages = sum((len(p) + 1 + PAGE - 1) // PAGE for p in prompts)
        state.update(specs=specs, pages=pages, pool=core.PagePool(pages, PAGE), slots=core.SlotPool(len(specs)) if eng.slots else None, make=core.Batch)
        for t in _cache(state):
            t.zero_()
        return state
    batch = core.Batch(seed, eng.pool, eng.slots)
    if not batch.add_prompts(specs, False):
        raise MemoryError("out of memory: no free pages for another state")
    before = [a for a, _ in reqs]
    if case["model"] == "llama3_8b":
        pages = torch.tensor([p for s in batch.seqs for p in s.pages], device="cuda")
        for l in range(LLAMA["layers"]):
            eng.kv[l].index_copy_(0, pages, _cached_llama(case, seed, l, pages.numel()))
        batch.advance(before)
    else:
        eng.step(batch, before)         # the contexts run through the model, which leaves caches and recurrent states
    state.update(batch=batch, counts=[b for _, b in reqs], back=[-b for _, b in reqs], want=[[b - 1] for _, b in reqs])
    return state


def _cache(state):
    """The part of the engine's cache that prompts fill: pages, and recurrent states."""
    eng, pages, n = state["engine"], state["pages"], len(state["specs"])
    if state["case"]["model"] == "llama3_8b":
        return [eng.kv[:, :pages]]
    out = []
    for i, r in enumerate(eng.cache.runs):
        if r.kv is not None and "kv_from" not in HYBRID[state["case"]["model"]]["layers"][i]["mixer"]:
            parts = [r.kv] if isinstance(r.kv, torch.Tensor) else [r.kv.pool] if hasattr(r.kv, "pool") else list(r.kv)
            out += [t[:pages] for t in parts]
        out += [t[:n] for t in (r.state, r.hist, r.mix_hist, r.shift) if t is not None]
    return out


def run(state):
    eng = state["engine"]
    if state["case"]["pass"] == "prefill":
        batch = state["make"](0, state["pool"], state["slots"])
        batch.add_prompts(state["specs"])
        eng.prefill(batch)
        out = {"logits": eng.runner.logits[:len(state["specs"])], "cache": _cache(state)}
        batch.clear()
        return out
    logits = eng.step(state["batch"], state["counts"], state["want"])
    state["batch"].advance(state["back"])       # back to where it was: the next pass is the same step
    return {"logits": logits}


# ---------------------------------------------------------------------------------------------------------- what a pass cannot do without
def _pairs(reqs, window=0, chunked=False, keep=0):
    """(visible keys of all queries, distinct keys read) of all requests."""
    pairs = keys = 0
    for a, b in reqs:
        if not window:
            pairs += b * a + b * (b + 1) // 2
            keys += a
            continue
        if chunked:
            pairs += sum(i % window + 1 for i in range(a, a + b))
            keys += a % window
        else:
            pairs += sum(min(i + 1, window) + (min(keep, i + 1 - window) if i + 1 > window else 0) for i in range(a, a + b))
            keys += min(a, window + keep)
    return pairs, keys


def work(case):
    reqs = _requests(case)
    T, n = sum(b for _, b in reqs), len(reqs)
    if case["model"] == "llama3_8b":
        c = LLAMA
        per_layer = sum(math.prod(s) for name, s in _llama_shapes() if name.startswith("layers.0."))
        pairs, keys = _pairs(reqs)
        kv = 2 * c["kv_heads"] * c["dim"] * c["layers"]
        weights = per_layer * c["layers"] + c["hidden"] * (c["vocab"] + 1)
        return {"bytes": 2 * (weights + T * c["hidden"] + kv * (keys + T)) + (2 if case["pass"] == "prefill" else 4) * n * c["vocab"],
                "flops": 2 * T * per_layer * c["layers"] + 2 * n * c["hidden"] * c["vocab"] + 4 * pairs * c["heads"] * c["dim"] * c["layers"]}
    c = HYBRID[case["model"]]
    H, V = c["width"], c["vocab"]
    read, flops, cache = H * V, 2 * n * H * V, 0
    for L in c["layers"]:
        m, f, kind = L["mixer"], L["mlp"], L["type"]
        dense, state = 0, 0
        for a in [m] if kind == "attention" else [m["left"]] if kind == "parallel" else []:
            own = "kv_from" not in a
            dense += H * a["heads"] * (a["dim"] + a["vdim"]) + own * H * a["kv_heads"] * (a["dim"] + (c["architecture"] != "Fafudra") * a["vdim"])
            pairs, keys = _pairs(reqs, a.get("mask", {}).get("size", 0), kind == "parallel", a.get("mask", {}).get("keep_first", 0))
            cache += own * 2 * (keys + T) * a["kv_heads"] * (a["dim"] + a["vdim"])
            flops += 2 * pairs * a["heads"] * (a["dim"] + a["vdim"])
        if kind == "parallel":
            b = m["right"]
            inner = b["heads"] * b["vdim"]
            dense += H * (2 * inner + 2 * b["groups"] * b["state"] + b["heads"]) + inner * H
            state = inner * b["state"]
        elif kind == "latent_attention":
            width = m["kv_rank"] + m["rot_dim"]
            dense += H * (m["q_rank"] + width) + m["q_rank"] * m["heads"] * (m["dim"] + m["rot_dim"]) + m["kv_rank"] * m["heads"] * (m["dim"] + m["vdim"]) + m["heads"] * m["vdim"] * H
            pairs, keys = _pairs(reqs, m.get("mask", {}).get("size", 0))
            cache += 2 * (keys + T) * width
            flops += 2 * pairs * m["heads"] * (m["dim"] + m["rot_dim"] + m["vdim"])
        elif kind == "gla":
            dense += H * m["heads"] * 2 * (m["dim"] + m["vdim"]) + H * m["rank"] + m["rank"] * m["heads"] * m["dim"] + m["heads"] * m["vdim"] * H
            state = m["heads"] * m["dim"] * m["vdim"]
        elif kind == "rglru":
            dense += 3 * H * m["width"] + 2 * m["width"] ** 2 // m["blocks"]
            state = m["width"]
        elif kind == "wkv":
            w = m["heads"] * m["dim"]
            dense += 5 * H * w + m["rank"] * (H + w)
            state = w * m["dim"]
        flops += 4 * T * state
        cache += 4 * state * (n + sum(1 for a, _ in reqs if a))     # written, and read where a request goes on
        if f and f["kind"] == "dense":
            dense += 3 * H * f["ff"]
        elif f:
            r, mats = f["router"], 3 if c["architecture"] == "Vofidra" else 2
            outputs, one = r["experts"] + r.get("identity", 0), mats * H * f["expert"]["ff"]
            shared = 2 * H * f["shared"]["ff"] if f.get("shared") else 0
            dense += H * outputs + shared
            read += r["experts"] * (1 - (1 - r["top"] / outputs) ** T) * one            # experts that some token chooses
            flops += 2 * T * r["top"] * r["experts"] / outputs * one
        read, flops = read + dense, flops + 2 * T * dense
    return {"bytes": 2 * (read + T * H) + cache + 4 * n * V, "flops": flops}


def tolerance(case):
    # 16-bit operands and activations between 8 to 32 layers, sums of 32 bits.  Measured against 64 bits, relative: logits 0.019 in
    # bfloat16 and 0.0024 in float16 (llama3_8b), 0.003 to 0.02 for the other designs' logits and caches.  Another order of the
    # same sums turns some of these roundings the other way: two such runs of one decode step differed by 0.01.
    if case["dtype"] == "float16":
        return {"rel": 0.01, "max": 0.3}
    return {"rel": 0.03, "max": 0.8}


# ---------------------------------------------------------------------------------------------------------- in 64 bits
class _Rows:
    """Rows of all requests, one after the other: `full`: every token from the first on, else those of the pass alone."""

    def __init__(self, case, seed, full):
        reqs, prompts = _requests(case), _prompts(case, seed)
        self.lens = [(a + b) if full else b for a, b in reqs]
        self.before = [0 if full else a for a, _ in reqs]
        self.first = [sum(self.lens[:i]) for i in range(len(reqs))]
        self.ids = torch.tensor([t for p, k in zip(prompts, self.lens) for t in p[len(p) - k:]], device="cuda")
        self.pos = torch.cat([torch.arange(a, a + k, device="cuda") for a, k in zip(self.before, self.lens)])
        self.last = torch.tensor([f + k - 1 for f, k in zip(self.first, self.lens)], device="cuda")
        self.new = reqs

    def of(self, i, x):
        return x[self.first[i]:self.first[i] + self.lens[i]]

    def paged(self, x):
        """Rows as the cache holds them: [pages, page, ...], with a place for one more token of every request."""
        out = []
        for i, n in enumerate(self.lens):
            rows = self.of(i, x)
            pad = (n + 1 + PAGE - 1) // PAGE * PAGE - n
            out.append(torch.cat([rows, rows.new_zeros(pad, *rows.shape[1:])]).view(-1, PAGE, *rows.shape[1:]))
        return torch.cat(out)


def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _turn(x, pos, freqs, interleaved, gain=1.0):
    """x [T, heads, d]: pairs of the first dimensions, neighbours or halves, turn by pos * freq."""
    n = freqs.numel()
    a = pos.double()[:, None] * freqs
    c, s = (a.cos() * gain)[:, None], (a.sin() * gain)[:, None]
    out = x.clone()
    iu = slice(0, 2 * n, 2) if interleaved else slice(0, n)
    iv = slice(1, 2 * n, 2) if interleaved else slice(n, 2 * n)
    u, v = x[..., iu], x[..., iv]
    out[..., iu], out[..., iv] = u * c - v * s, v * c + u * s
    return out


def _freqs(dims, base, scaling=None):
    f = [base ** (-2.0 * i / dims) for i in range(dims // 2)]
    if scaling:
        at = lambda turns: dims * math.log(scaling["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(base))
        lo, hi = max(math.floor(at(scaling["fast"])), 0), min(math.ceil(at(scaling["slow"])), dims - 1)
        ramp = [min(max((i - lo) / max(hi - lo, 0.001), 0.0), 1.0) for i in range(dims // 2)]
        f = [x / scaling["factor"] * t + x * (1.0 - t) for x, t in zip(f, ramp)]
    return torch.tensor(f, device="cuda", dtype=torch.float64)


def _attend(q, k, v, scale, first=0, see=None, bias=None, cap=0.0, sink=None, sigmoid=None):
    """q [T, H, d] of positions first, first + 1, ..; k [S, G, d], v [S, G, n] of positions 0, 1, ..: [T, H, n]."""
    T, H, d = q.shape
    S, G, n = v.shape
    out = torch.empty(T, H, n, device="cuda", dtype=torch.float64)
    kt = k.permute(1, 2, 0)[:, None]
    vt = v.permute(1, 0, 2)[:, None]
    step = max(1, min(T, (1 << 28) // (H * S)))
    j = torch.arange(S, device="cuda")[None, :]
    for t in range(0, T, step):
        rows = q[t:t + step]
        i = torch.arange(first + t, first + t + len(rows), device="cuda")[:, None]
        s = (rows.permute(1, 0, 2).reshape(G, H // G, len(rows), d) @ kt).reshape(H, len(rows), S) * scale
        if bias is not None:
            s = s + bias(i - j)
        if cap:
            s = cap * torch.tanh(s / cap)
        ok = j <= i
        if see is not None:
            ok = ok & see(i, j)
        if sigmoid is not None:
            w = torch.sigmoid(s + sigmoid[:, None, None]) * ok
        else:
            s = s.masked_fill(~ok, float("-inf"))
            if sink is not None:
                s = torch.cat([s, sink[:, None, None].expand(H, len(rows), 1)], -1)
            w = torch.softmax(s, -1)[..., :S]
        out[t:t + step] = (w.reshape(G, H // G, len(rows), S) @ vt).reshape(H, len(rows), n).permute(1, 0, 2)
    return out


def _linear(x, w, out=None):
    """x @ w in 64 bits, a part of the rows at a time."""
    w = w.double()
    return torch.cat([p @ w for p in x.split(8192)])


def _llama_exact(case, seed):
    c, dt = LLAMA, DTYPES[case["dtype"]]
    rows, shapes = _Rows(case, seed, False), _llama_shapes()
    index = {n: i for i, (n, _) in enumerate(shapes)}
    w = lambda n: _llama_weight(index[n], n, shapes[index[n]][1], dt)
    H, G, d, ff = c["heads"], c["kv_heads"], c["dim"], c["inter"]
    x = w("embed")[rows.ids].double()
    T, freqs, caches = x.shape[0], _freqs(d, c["theta"]), []
    pages = [(a + b + PAGE - 1) // PAGE for a, b in rows.new]
    for l in range(c["layers"]):
        p = f"layers.{l}."
        h = _rms(x, c["eps"]) * w(p + "input_ln").double()
        q, k, v = _linear(h, w(p + "qkv")).split([H * d, G * d, G * d], -1)
        q, k, v = _turn(q.view(T, H, d), rows.pos, freqs, False), _turn(k.view(T, G, d), rows.pos, freqs, False), v.view(T, G, d)
        held = _cached_llama(case, seed, l, sum(pages)) if case["pass"] != "prefill" else None
        att = torch.empty(T, H, d, device="cuda", dtype=torch.float64)
        for i, (a, b) in enumerate(rows.new):
            kk, vv = rows.of(i, k), rows.of(i, v)
            if a:
                own = held[sum(pages[:i]):sum(pages[:i + 1])].double()
                kk, vv = (torch.cat([own[:, s].reshape(-1, G, d)[:a], t]) for s, t in ((0, kk), (1, vv)))
            rows.of(i, att).copy_(_attend(rows.of(i, q), kk, vv, d ** -0.5, a))
        x = x + _linear(att.view(T, H * d), w(p + "o"))
        h = _rms(x, c["eps"]) * w(p + "post_ln").double()
        gu, down = w(p + "gate_up").double(), w(p + "down").double()
        for t in range(0, T, 4096):
            g, u = (h[t:t + 4096] @ gu).split(ff, -1)
            x[t:t + 4096] += (torch.nn.functional.silu(g) * u) @ down
        if case["pass"] == "prefill":
            caches.append(torch.stack([rows.paged(k), rows.paged(v)], 1).float())
    logits = (_rms(x[rows.last], c["eps"]) * w("final_norm").double()) @ w("lm_head").double()
    return {"logits": logits, "cache": [torch.stack(caches)]} if caches else {"logits": logits}


def _scan(rows, step, n_state, outs):
    """Runs `step(state, t, index of the rows at that place, which requests)` over the places of all requests side by side; returns
    the states at the end and the outputs [T, ...]."""
    first = torch.tensor(rows.first, device="cuda")
    order = sorted(range(len(rows.lens)), key=lambda i: -rows.lens[i])      # longest first: those that go on are a prefix
    lens = [rows.lens[i] for i in order]
    first = first[torch.tensor(order, device="cuda")]
    state = torch.zeros(len(order), *n_state, device="cuda", dtype=torch.float64)
    live = len(order)
    for t in range(lens[0]):
        while lens[live - 1] <= t:
            live -= 1
        at = first[:live] + t
        outs[at] = step(state[:live], at)
    return state[torch.tensor([order.index(i) for i in range(len(order))], device="cuda")], outs


def _conv(x, w, pos):
    """Causal convolution of every request's rows: x [T, channels], w [channels, taps], the last column for the current row."""
    taps, out = w.shape[1], x * w[:, -1]
    for back in range(1, taps):
        if back < x.shape[0]:
            out[back:] += x[:-back] * w[:, taps - 1 - back] * (pos[back:, None] >= back)
    return out


def _gla(h, w, m, eps, rows):
    T, H, dk, dv = h.shape[0], m["heads"], m["dim"], m["vdim"]
    q, k, v = (_linear(h, w(n).t()).view(T, H, -1) for n in "qkv")
    z = (_linear(_linear(h, w("a1").t()), w("a2").t()) + w("a2.b").double()).view(T, H, dk)
    alpha = torch.sigmoid(z) ** (1.0 / m["tau"])

    def step(S, at):
        S.mul_(alpha[at][..., None]).addcmul_(k[at][..., None], v[at][:, :, None])
        return (S * q[at][..., None]).sum(2)
    state, o = _scan(rows, step, (H, dk, dv), torch.empty(T, H, dv, device="cuda", dtype=torch.float64))
    o = _rms(o * dk ** -0.5, eps) * w("norm").double()
    return _linear(o.reshape(T, -1) * torch.nn.functional.silu(_linear(h, w("g").t())), w("o").t()), [state]


def _rglru(h, w, m, rows):
    T, W, nb = h.shape[0], m["width"], m["blocks"]
    y = torch.nn.functional.gelu(_linear(h, w("y").t()) + w("y.b").double(), approximate="tanh")
    x = _linear(h, w("x").t()) + w("x.b").double()
    u = _conv(x, w("conv").double(), rows.pos) + w("conv.b").double()
    gate = lambda n: torch.sigmoid(torch.einsum("tbi,boi->tbo", u.view(T, nb, -1), w(n).double()) + w(n + ".b").double()).reshape(T, W)
    a = torch.exp(-8.0 * gate("ra") * torch.nn.functional.softplus(w("lam").double(), threshold=1e9))
    b = torch.sqrt(1.0 - a * a) * gate("ri") * u

    def step(S, at):
        return S.mul_(a[at]).add_(b[at])
    state, o = _scan(rows, step, (W,), torch.empty_like(u))
    return _linear(o * y, w("o").t()), [state, None]


def _wkv(h, w, m, eps, rows):
    T, H, n = h.shape[0], m["heads"], m["dim"]
    prev = torch.cat([torch.zeros_like(h[:1]), h[:-1]]) * (rows.pos > 0)[:, None]
    mixed = lambda s: h + (prev - h) * w("mu." + s).double()
    r, k, v = (_linear(mixed(s), w(s).t()).view(T, H, n) for s in "rkv")
    gate = torch.nn.functional.silu(_linear(mixed("g"), w("g").t()))
    z = _linear(torch.tanh(_linear(mixed("w"), w("w1").t())), w("w2").t()) + w("w0").double()
    decay, u = torch.exp(-torch.exp(z)).view(T, H, n), w("u").double()

    def step(S, at):
        kv = k[at][..., None] * v[at][:, :, None]
        o = ((S + u[..., None] * kv) * r[at][..., None]).sum(2)
        S.mul_(decay[at][..., None]).add_(kv)
        return o
    state, o = _scan(rows, step, (H, n, n), torch.empty(T, H, n, device="cuda", dtype=torch.float64))
    return _linear((_rms(o, eps).reshape(T, -1) * w("norm").double()) * gate, w("o").t()), [state]


def _latent(h, w, m, eps, rows, gated):
    T, H, d, r, nv, rank = h.shape[0], m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
    freqs = _freqs(r, m["rot"]["base"])
    q = _linear(_rms(_linear(h, w("dq").t()), eps) * w("dq.norm").double(), w("uq").t()).view(T, H, d + r)
    ckv = _linear(h, w("dkv").t())
    c, kr = _rms(ckv[:, :rank], eps) * w("dkv.norm").double(), _turn(ckv[:, None, rank:], rows.pos, freqs, not gated)
    k, v = _linear(c, w("uk").t()).view(T, H, d), _linear(c, w("uv").t()).view(T, H, nv)
    q = torch.cat([q[..., :d], _turn(q[..., d:], rows.pos, freqs, not gated)], -1)
    k = torch.cat([k, kr.expand(T, H, r)], -1)
    window = m.get("mask", {}).get("size", 1 << 40)
    sink = None if gated else w("sink").double()
    o = torch.cat([_attend(rows.of(i, q), rows.of(i, k), rows.of(i, v), m["scale"], see=lambda i, j: i - j < window, sink=sink)
                   for i in range(len(rows.lens))])
    if gated:
        o = o * torch.sigmoid(_linear(h, w("g").t()))[..., None]
    return _linear(o.reshape(T, -1), w("o").t()), [rows.paged(torch.cat([c, kr[:, 0]], -1)[:, None])]


def _ssd(h, w, m, eps, rows):
    T, H, P, N, G = h.shape[0], m["heads"], m["vdim"], m["state"], m["groups"]
    inner = H * P
    z, xbc, dt = torch.split(_linear(h, w("in").t()), [inner, inner + 2 * G * N, H], -1)
    xbc = torch.nn.functional.silu(_conv(xbc, w("conv").double(), rows.pos) + w("conv.b").double())
    x, B, C = torch.split(xbc, [inner, G * N, G * N], -1)
    x, B, C = x.reshape(T, H, P), B.reshape(T, G, N).repeat_interleave(H // G, 1), C.reshape(T, G, N).repeat_interleave(H // G, 1)
    dt = torch.nn.functional.softplus(dt + w("dt_bias").double(), threshold=1e9)
    decay, skip = torch.exp(-torch.exp(w("A_log").double()) * dt), w("D").double()[:, None]

    def step(S, at):
        S.mul_(decay[at][..., None, None]).add_((dt[at][..., None] * B[at])[..., None] * x[at][:, :, None])
        return (S * C[at][..., None]).sum(2) + skip * x[at]
    state, y = _scan(rows, step, (H, N, P), torch.empty(T, H, P, device="cuda", dtype=torch.float64))
    y = y.reshape(T, -1) * torch.nn.functional.silu(z)
    y = _rms(y.view(T, m["norm_groups"], -1), eps).reshape(T, -1) * w("norm").double()
    return _linear(y, w("o").t()), [state, None]


def _attention(h, w, m, eps, rows, kind, shared):
    T, H, G, d = h.shape[0], m["heads"], m["kv_heads"], m["dim"]
    proj = lambda n: _linear(h, w(n).t()) + (w(n + ".b").double() if kind == "Komulorn" else 0.0)
    q, more = proj("q").view(T, H, d), {}
    if shared is None:
        k = proj("k").view(T, G, d)
        v = k if kind == "Fafudra" else proj("v").view(T, G, m["vdim"])
    if kind == "Vofidra":
        q, k = _rms(q, eps) * w("q.norm").double(), _rms(k, eps) * w("k.norm").double()
        t = m["q_temp"]
        q = q * (1.0 + t["coef"] * torch.log((rows.pos + 1).div(t["every"], rounding_mode="floor").double() + 1.0))[:, None, None]
        rel, half, far, n = w("rel").double(), m["rows"] // 2, m["bias_max"], m["rows"]
        row = [i if i < half else min(n - 1, half + math.floor(math.log(i / half) / math.log(far / half) * (n - half))) for i in range(max(rows.lens))]
        table = rel[torch.tensor(row, device="cuda")].t()
        more["bias"] = lambda dist: table[:, dist.clamp(min=0)]
    else:
        if kind == "Norusun":
            q, k = ((_rms(x.reshape(T, -1), eps) * w(n).double()).view(x.shape) for x, n in ((q, "q.norm"), (k, "k.norm")))
        rot = m["rot"]
        f, inter = _freqs(rot["dims"], rot["base"], rot.get("scaling")), kind == "Fafudra"
        gain = 0.1 * math.log(rot["scaling"]["factor"]) + 1.0 if "scaling" in rot else 1.0
        q = _turn(q, rows.pos, f, inter, gain)
        if shared is None:
            k = _turn(k, rows.pos, f, inter, gain)
    k, v = shared or (k, v)
    if kind == "Fafudra":
        size, keep = m["mask"]["size"], m["mask"]["keep_first"]
        more.update(cap=m["softcap"], sink=w("sink").double(), see=lambda i, j: (i - j < size) | (j < keep))
    elif kind == "Norusun":
        size = m["mask"]["size"]
        more.update(sigmoid=w("pb").double(), see=lambda i, j: i // size == j // size)
    o = torch.cat([_attend(rows.of(i, q), rows.of(i, k), rows.of(i, v), m["scale"], **more) for i in range(len(rows.lens))])
    if kind == "Komulorn":
        o = o * torch.sigmoid(_linear(h, w("g").t()))[..., None]
    if shared is not None:
        held = []
    elif m["vdim"] == d:
        held = [torch.stack([rows.paged(k), rows.paged(v)], 1)]
    else:
        held = [rows.paged(k), rows.paged(v)]
    return _linear(o.reshape(T, -1), w("o").t()), held, (k, v)


def _experts(h, w, f, kind):
    r, out = f["router"], torch.zeros_like(h)
    z = _linear(h, w("router").t())
    if kind == "Komulorn":
        val, idx = torch.topk(torch.sigmoid(z), r["top"], dim=-1)
    else:
        s = torch.softmax(z, -1)
        choice = s + w("correction").double()
        per = choice.view(len(h), r["groups"]["count"], -1)
        best = per.max(-1).values.topk(r["groups"]["keep"], dim=-1).indices
        keep = torch.zeros(per.shape[:2], dtype=torch.bool, device="cuda").scatter_(1, best, True)
        idx = per.masked_fill(~keep[..., None], float("-inf")).view_as(choice).topk(r["top"], dim=-1).indices
        val = s.gather(1, idx)
        val = val / (val.sum(-1, keepdim=True) + 1e-20)
    for e in range(z.shape[1]):
        t, k = (idx == e).nonzero(as_tuple=True)
        wt, x = val[t, k][:, None], h[t]
        if e >= r["experts"]:
            out[t] += wt * x
        elif len(t) and kind == "Komulorn":
            out[t] += torch.relu((wt * x) @ w(f"e{e}.up").double().t()).square() @ w(f"e{e}.down").double().t()
        elif len(t):
            g, u = x @ w(f"e{e}.gate").double().t(), x @ w(f"e{e}.up").double().t()
            out[t] += wt * ((torch.nn.functional.silu(g) * u) @ w(f"e{e}.down").double().t())
    if f.get("shared"):
        out += torch.relu(h @ w("shared.up").double().t()).square() @ w("shared.down").double().t() * torch.sigmoid(h @ w("shared.sg").double().t())
    return out


def _feed_forward(h, w, f, kind):
    out = []
    gate, up, down = (w(n).double().t() for n in ("gate", "up", "down"))
    for x in h.split(4096):
        g, u = x @ gate, x @ up
        if kind == "Norusun":
            g, u = (g + w("gate.b").double()).clamp(max=f["limit"]), (u + w("up.b").double()).clamp(-f["limit"], f["limit"])
            out.append((g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ down + w("down.b").double())
        else:
            out.append((torch.nn.functional.silu(g) * u) @ down)
    return torch.cat(out)


def _hybrid_exact(case, seed):
    c, rows = HYBRID[case["model"]], _Rows(case, seed, True)
    kind, eps, S, weights, caches, kvs = c["architecture"], c["norm"]["eps"], c.get("streams", 0), _hybrid_weights(c), [], {}
    w = weights.__getitem__

    def norm(x, name):
        if kind == "Vofidra":
            return torch.tanh(w(name + ".alpha").double() * x) * w(name).double() + w(name + ".b").double()
        return _rms(x, eps) * (w(name).double() + (1.0 if kind == "Fafudra" else 0.0))

    def mixer(i, L, h):
        mix, m = (lambda n: w(f"l{i}.mix.{n}")), L["mixer"]
        if L["type"] == "attention":
            y, held, kvs[i] = _attention(h, mix, m, eps, rows, kind, kvs.get(m.get("kv_from")))
        elif L["type"] == "latent_attention":
            y, held = _latent(h, mix, m, eps, rows, kind == "Vofidra")
        elif L["type"] == "parallel":
            a, held, _ = _attention(h, lambda n: mix("left." + n), m["left"], eps, rows, kind, None)
            b, more = _ssd(h, lambda n: mix("right." + n), m["right"], eps, rows)
            y, held = 0.5 * (_rms(a, eps) * mix("left.out").double() + _rms(b, eps) * mix("right.out").double()), held + more
        else:
            y, held = {"gla": lambda: _gla(h, mix, m, eps, rows), "rglru": lambda: _rglru(h, mix, m, rows), "wkv": lambda: _wkv(h, mix, m, eps, rows)}[L["type"]]()
        caches.extend(held + ([None] if c.get("canon") else []) + ([None] if L["type"] == "wkv" else []))
        return y

    x = w("embed")[rows.ids].double()
    xs = x[None].repeat(S, 1, 1) if S else None
    for i, L in enumerate(c["layers"]):
        mlp = lambda n: w(f"l{i}.mlp.{n}")
        forward = lambda h: _feed_forward(h, mlp, L["mlp"], kind) if L["mlp"]["kind"] == "dense" else _experts(h, mlp, L["mlp"], kind)
        if kind == "Fafudra":
            h = norm(x, f"l{i}.norm1")
            x = x + c["residual_mult"] * (mixer(i, L, h) + forward(h))
            continue
        for q in (1, 2) if L["mlp"] else (1,):
            h = norm(torch.einsum("s,stw->tw", w(f"l{i}.hc{q}.in").double(), xs) if S else x, f"l{i}.norm{q}")
            if q == 1 and c.get("canon"):
                h = h + _conv(h, w(f"l{i}.canon1").double(), rows.pos)
            y = mixer(i, L, h) if q == 1 else forward(h)
            if S:
                xs = torch.einsum("su,stw->utw", w(f"l{i}.hc{q}.mix").double(), xs) + w(f"l{i}.hc{q}.out").double()[:, None, None] * y
            else:
                x = x + y
    x = xs.sum(0)[rows.last] if S else x[rows.last]
    z = norm(x, "final.norm") @ w("embed" if kind == "Fafudra" else "head").double().t()
    if c.get("logit_softcap"):
        z = c["logit_softcap"] * torch.tanh(z / c["logit_softcap"])
    return {"logits": z, "cache": caches} if case["pass"] == "prefill" else {"logits": z}


@torch.no_grad()
def exact(case, seed):
    if case["model"] == "llama3_8b":
        return _llama_exact(case, seed)
    if sum(a + b for a, b in _requests(case)) > 40000:
        return None
    return _hybrid_exact(case, seed)
