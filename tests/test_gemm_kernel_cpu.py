"""Which kernel runs a product that carries no hint (no GPU; needs the built library)."""
import random

import pytest

from blitz_scale_b200 import ops

TILED, STREAM, PAIR, WIDE, QUAD = 0, 1, 2, 3, 4
STORE, ADD, SILU, STORE32, F32, CAP, GLU = 0, 1, 2, 4, 5, 6, 7

# the kernel that runs where no hint is given: what is one round of 33 clusters of four, and K beyond 512, goes to those
KERNEL = [
    ((1, 4096, 4096, STORE, 1), STREAM), ((128, 4096, 4096, ADD, 1), STREAM), ((129, 4096, 4096, ADD, 1), QUAD), ((256, 6144, 4096, STORE, 1), WIDE),
    ((136, 2048, 14336, STORE, 1), STREAM), ((256, 6144, 8192, ADD, 1), PAIR), ((193, 14336, 4096, SILU, 1), WIDE), ((192, 14336, 4096, SILU, 1), STREAM),
    ((300, 2048, 4096, STORE, 1), QUAD), ((300, 2176, 4096, STORE, 1), TILED), ((300, 2048, 520, ADD, 1), QUAD), ((300, 2048, 512, ADD, 1), WIDE),
    ((300, 2048, 256, STORE, 1), WIDE), ((3000, 128, 2048, STORE, 1), QUAD), ((8448, 128, 576, STORE, 1), QUAD), ((8449, 128, 576, STORE, 1), TILED),
    ((1000, 1024, 2048, F32, 1), QUAD), ((1000, 1024, 2048, SILU, 1), WIDE), ((384, 2816, 2048, SILU, 1), TILED), ((300, 56, 4096, STORE, 1), TILED),
    ((300, 256, 192, STORE, 16), TILED), ((1574, 4096, 4096, ADD, 1), WIDE), ((300, 5632, 2048, SILU, 1), TILED),
]


@pytest.mark.skipif(not ops.available(), reason="kernel library not built")
@pytest.mark.parametrize("shape,want", KERNEL)
def test_kernel(shape, want):
    assert ops.lib().blitz_gemm_kernel(*shape) == want


@pytest.mark.skipif(not ops.available(), reason="kernel library not built")
def test_the_kernel_named_takes_the_product():
    L, rng = ops.lib(), random.Random(3)
    supported = {STREAM: lambda M, N, K, e, g: g == 1 and L.blitz_gemm_decode_supported(M, N, K, 0, e),
                 PAIR: lambda M, N, K, e, g: g == 1 and L.blitz_gemm_pair_supported(M, N, K, 0, e),
                 WIDE: lambda M, N, K, e, g: L.blitz_gemm_wide_supported(M, N, K, 0, e, g),
                 QUAD: lambda M, N, K, e, g: g == 1 and L.blitz_gemm_quad_supported(M, N, K, 0, e), TILED: lambda *a: True}
    some = lambda top: 8 * round(2 ** rng.uniform(0, top))
    used = set()
    for _ in range(50000):
        shape = (round(2 ** rng.uniform(0, 14)), some(14), some(11), rng.choice([STORE, ADD, SILU, STORE32, F32, CAP, GLU]), rng.choice([1, 1, 1, 8]))
        kernel = L.blitz_gemm_kernel(*shape)
        assert supported[kernel](*shape), (shape, kernel)
        used.add(kernel)
    assert used == set(supported)
