"""The products of many rows (CTA pairs, 256 x 256 tiles) at the edges of their tiles against fp32 products of the same operands."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"

# rows, columns, depth: below and behind a tile's edge, one K block and less, last rounds of halved and of whole tiles, columns that do
# not come in slabs of 64
SIZES = [(1, 64, 8), (257, 64, 64), (300, 136, 72), (512, 512, 512), (777, 1000, 1032), (1574, 6144, 256), (256, 14336, 256), (4999, 1032, 136)]


@pytest.mark.parametrize("M,N,K", SIZES)
@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
def test_epilogues(M, N, K, dt):
    from blitz_scale_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(M + N)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g).to(dt)
    a, w, r = rnd(M, K + 8)[:, :K], (rnd(K, N).float() * K ** -0.5).to(dt), rnd(M, N)
    ref = a.float() @ w.float()
    unit = 2.0 ** -8 if dt == torch.bfloat16 else 2.0 ** -11

    def near(got, want, rel):    # one rounding of the result, and 32-bit sums in another order
        assert float(((got.float() - want).abs() - rel * want.abs()).max()) <= 2e-5 * K ** 0.5
    run = lambda out, **kw: ops.gemm(a, w, out=out, wide_path=True, **kw)
    near(run(torch.full((M, N), 7.0, dtype=dt, device=DEV)), ref, unit)
    both = r.clone()
    near(run(both, residual=both, epilogue="add"), ref + r.float(), unit)
    near(run(torch.zeros(M, N, device=DEV)), ref, 1e-5)
    near(run(torch.ones(M, N, device=DEV), epilogue="axpy", alpha=0.5), 1 + 0.5 * ref, 1e-5)
    near(run(torch.zeros(M, N, device=DEV), epilogue="softcap", alpha=2.0), 2 * torch.tanh(ref / 2), 1e-5)
    if N % 16 == 0 and N >= 128:
        gate, up = ref[:, :N // 2], ref[:, N // 2:]
        near(run(None, epilogue="silu_mul"), torch.nn.functional.silu(gate) * up, 2 * unit)
        bias = rnd(N)
        gb, ub = (gate + bias[:N // 2].float()).clamp(max=1.5), (up + bias[N // 2:].float()).clamp(-1.5, 1.5)
        near(run(None, epilogue="clamp_glu", alpha=1.5, beta=1.7, bias=bias), gb * torch.sigmoid(1.7 * gb) * (ub + 1), 2 * unit)
    ops.check_status()


@pytest.mark.parametrize("M", [257, 700])
@pytest.mark.parametrize("f32", [False, True])
def test_diagonal_blocks(M, f32):
    from blitz_scale_b200 import ops
    G, K, N = 4, 192, 320
    a = torch.randn(M, G * (K + 8), device=DEV).to(torch.bfloat16)
    w = (torch.randn(G * K, N, device=DEV) * K ** -0.5).to(torch.bfloat16)
    out = torch.full((M, G * (N + 16)), 7.0, dtype=torch.float32 if f32 else torch.bfloat16, device=DEV)
    ops.gemm(a, w, out=out, groups=G, a_step=K + 8, out_step=N + 16, wide_path=True)
    ops.check_status()
    for i in range(G):
        want = a[:, i * (K + 8):i * (K + 8) + K].float() @ w[i * K:(i + 1) * K].float()
        got = out[:, i * (N + 16):(i + 1) * (N + 16)]
        assert float(((got[:, :N].float() - want).abs() - (1e-5 if f32 else 2.0 ** -8) * want.abs()).max()) <= 2e-5 * K ** 0.5
        assert bool((got[:, N:] == 7.0).all())


@pytest.mark.parametrize("M", [129, 300, 1574])
def test_silu_of_large_negative_gates(M):
    """Denominators beyond 2^126, where an approximate division answers zero."""
    from blitz_scale_b200 import ops
    N, K = 192, 64
    gates = torch.cat([torch.linspace(-88.5, -80.0, 96), torch.linspace(-20.0, 20.0, 96)]).to(torch.bfloat16)
    w = torch.zeros(K, 2 * N, dtype=torch.bfloat16, device=DEV)
    w[0, :N], w[0, N:] = gates.to(DEV), 2.0 ** 100
    a = torch.zeros(M, K, dtype=torch.bfloat16, device=DEV)
    a[:, 0] = 1
    got = ops.gemm(a, w, epilogue="silu_mul", wide_path=True).double()
    g = gates.double().to(DEV)
    want = (g / (1 + torch.exp(-g)) * 2.0 ** 100).expand(M, N)
    # one rounding to bf16; the exponential of fp32 numbers is off by 2 + 1.16 |x| units of fp32
    assert bool(((got - want).abs() <= want.abs() * (2.0 ** -8 + 110 * 2.0 ** -23)).all())


# at the lines of the rule that chooses between this kernel and the tiled one (tests/test_gemm_choice_cpu.py), both sides
@pytest.mark.parametrize("M,N,K,epi", [(384, 6144, 136, "store"), (385, 6144, 136, "store"), (1024, 2304, 72, "add"), (1152, 2304, 72, "add"),
                                       (300, 9472, 64, "store"), (300, 9480, 64, "store"), (1300, 2048, 2048, "axpy"), (1300, 2048, 2056, "axpy")])
def test_default_dispatch(M, N, K, epi):
    from blitz_scale_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(M + K)
    a, w = torch.randn(M, K, device=DEV, generator=g).bfloat16(), (torch.randn(K, N, device=DEV, generator=g) * K ** -0.5).bfloat16()
    old = torch.randn(M, N, device=DEV, generator=g).to(torch.float32 if epi == "axpy" else torch.bfloat16)
    want = a.float() @ w.float() + (old.float() if epi != "store" else 0)
    out = ops.gemm(a, w, out=old.clone(), residual=old if epi == "add" else None, epilogue=epi)
    ops.check_status()
    # one rounding of the result, and 32-bit sums in another order
    assert float(((out.float() - want).abs() - (1e-5 if epi == "axpy" else 2.0 ** -8) * want.abs()).max()) <= 2e-5 * K ** 0.5


@pytest.mark.parametrize("M", [129, 144, 192, 193, 224, 225, 256])
@pytest.mark.parametrize("N,K,epi", [(1024, 1024, "store"), (2048, 2048, "add"), (6144, 4096, "store"), (6144, 8192, "add"), (9600, 576, "silu_mul"), (1088, 520, "silu_mul")])
def test_between_decode_batches_and_prompts(M, N, K, epi):
    """129 to 256 rows: whichever kernel takes them, against sums in 64 bits and the paired kernel."""
    from blitz_scale_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(M + N)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda").to(torch.bfloat16)
    a, b, res = r(M, K), r(K, 2 * N if epi == "silu_mul" else N) * K ** -0.5, r(M, N)
    acc = a.double() @ b.double()
    ref = torch.nn.functional.silu(acc[:, :N]) * acc[:, N:] if epi == "silu_mul" else acc + res.double() if epi == "add" else acc
    outs = []
    for kw in ({}, dict(pair_path=True)):
        out = res.clone()
        ops.gemm(a, b, out=out, epilogue=epi, static_b=True, **(dict(residual=out) if epi == "add" else {}), **kw)
        # one rounding of the output, and sums of K products of size K^-0.5 in fp32
        assert ((out.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-4).all(), kw
        outs.append(out)
    ops.check_status()
    used = ops.lib().blitz_gemm_few_rows(M, N, K, {"store": 0, "add": 1, "silu_mul": 2}[epi])
    assert used in (1, 2, 3, 4)
    if used == 2:
        assert torch.equal(*outs)
