"""Single tokens beside a portion, through decode attention or among the portion's tiles: the logits of whole prompts."""
import pytest
import torch

from hybrid_feed import Feed

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("apart", [True, False])
def test_singles(monkeypatch, apart):
    from blitz_scale_b200 import ops
    from blitz_scale_b200.runtime import engine
    torch.cuda.set_device(0)
    monkeypatch.setattr(engine, "singles_apart", lambda *a: apart)
    eng = engine.Engine("tiny_gpu", num_pages=128, page_size=16, max_batch=8, max_batch_tokens=512, seed=1)
    toks = torch.randint(0, 4096, (300,), generator=torch.Generator().manual_seed(8)).tolist()
    f = Feed(eng)
    f.step({0: toks})
    f.step({1: toks[:129], 2: toks[:20], 3: toks[:5]})
    f.step({1: toks[129:150], 2: toks[20:21], 3: toks[5:6]})
    f.step({1: toks[150:151], 2: toks[21:160], 3: toks[6:7]})
    f.step({1: toks[151:], 2: toks[160:161], 3: toks[7:140]})
    f.step({2: toks[161:], 3: toks[140:]})
    ops.check_status()
    whole = f.logits(0)
    for r in (1, 2, 3):
        err = (f.logits(r) - whole).pow(2).mean(-1).sqrt() / whole.pow(2).mean().sqrt()
        assert float(err.max()) < 3e-2, (r, float(err.max()))      # as for portions and single tokens elsewhere: bf16 roundings
