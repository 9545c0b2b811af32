"""A prompt longer than one forward pass takes is prefetched in chunks over the paged cache and gives the tokens of a
single pass."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model,lens", [("tiny_gpu", [1300, 40, 700, 513]), ("tiny_gpu_deep", [2100])])
def test_chunked_prefill_equals_single_pass(model, lens):
    import torch
    from blitz_scale_b200 import ops
    from blitz_scale_b200.runtime import core
    from blitz_scale_b200.runtime.engine import Engine
    torch.cuda.set_device(0)
    g = torch.Generator().manual_seed(3)
    prompts = [torch.randint(0, 4096, (n,), generator=g).tolist() for n in lens]
    outs = []
    for budget in (4096, 512):
        eng = Engine(model, num_pages=256, page_size=16, max_batch=8, max_batch_tokens=budget, seed=1, use_graphs=False)
        b = eng.new_batch(1, [core.SeqSpec(i, p, 6) for i, p in enumerate(prompts)])
        assert b is not None
        seqs = [[t] for t in eng.prefill(b)]
        logits = [eng.runner.logits[:len(lens)].float().clone()]
        for _ in range(4):
            for sq, t in zip(seqs, eng.decode(b)):
                sq.append(t)
            logits.append(eng.runner.logits[:len(lens)].float().clone())
        ops.check_status()
        outs.append((seqs, logits))
        b.clear()
        assert eng.pool.used_pages == 0
        del eng
        torch.cuda.empty_cache()
    (one, l1), (chunked, l2) = outs
    # the same attention in different tilings: logits agree closely; tokens are equal unless two candidates tie
    err = float((l1[0] - l2[0]).norm() / l1[0].norm())
    assert err < 2e-2, err
    ties = 0
    for r, (x, y) in enumerate(zip(one, chunked)):
        at = next((i for i, (a, c) in enumerate(zip(x, y)) if a != c), None)
        if at is None:
            continue
        # the passes before were of the same tokens: their logits agree as closely, and the two candidates are at most two units of
        # bf16 (2^-7 of the value at most) apart in both; what follows is another text
        ties += 1
        p, q = l1[at][r], l2[at][r]
        assert float((p - q).norm() / p.norm()) < 2e-2, (r, at)
        for row in (p, q):
            assert abs(float(row[x[at]] - row[y[at]])) <= 2 * 2 ** -7 * float(row.max()), (r, at, one, chunked)
    assert ties <= 1, (one, chunked)
