"""Which kernel takes a product: the rules that the library decides by (no GPU; needs the built library)."""
import random

import pytest

from blitz_scale_b200 import ops

TILED, STREAM, PAIR, WIDE, QUAD = 0, 1, 2, 3, 4
STORE, ADD, SILU, STORE32, F32, CAP, GLU = 0, 1, 2, 4, 5, 6, 7

# rows, columns, depth, epilogue, blocks -> kernel that a call with hints starts from, as measured on both sides of every line
FAMILY = [
    ((1, 4096, 4096, STORE, 1), STREAM), ((128, 4096, 4096, ADD, 1), STREAM), ((129, 4096, 4096, ADD, 1), PAIR), ((256, 6144, 4096, STORE, 1), PAIR),
    # a round of tiles of 128 x 128
    ((300, 2048, 4096, STORE, 1), TILED), ((257, 6144, 4096, STORE, 1), TILED), ((384, 6144, 4096, ADD, 1), TILED), ((400, 6144, 4096, STORE, 1), WIDE),
    ((2048, 1152, 8192, STORE, 1), TILED), ((1024, 2048, 2048, STORE, 1), TILED), ((900, 2048, 4096, F32, 1), TILED),
    ((512, 2560, 1024, ADD, 1), WIDE), ((1152, 2048, 1024, ADD, 1), TILED), ((1000, 1024, 2048, SILU, 1), WIDE), ((384, 2816, 2048, SILU, 1), TILED),
    ((6400, 136, 2048, STORE, 1), WIDE),
    # rows that fill a little more than one tile of 256
    ((300, 10240, 4096, STORE, 1), TILED), ((300, 5632, 2048, SILU, 1), TILED), ((300, 14336, 4096, SILU, 1), WIDE), ((300, 16384, 1024, STORE, 1), WIDE),
    # narrow blocks
    ((1000, 128, 512, STORE, 32), TILED), ((4096, 64, 512, STORE, 8), TILED), ((4096, 128, 512, STORE, 32), WIDE), ((1574, 64, 512, STORE, 32), TILED), ((2500, 64, 512, STORE, 32), WIDE), ((300, 256, 192, STORE, 16), TILED),
    ((600, 256, 128, STORE, 32), WIDE),
    # one round into fp32
    ((1290, 2048, 1024, F32, 1), TILED), ((1290, 2048, 4096, F32, 1), WIDE), ((2600, 2048, 1024, F32, 1), WIDE),
    ((1574, 4096, 4096, ADD, 1), WIDE), ((8192, 6144, 4096, STORE, 1), WIDE), ((8192, 14336, 4096, SILU, 1), WIDE),
]


@pytest.mark.skipif(not ops.available(), reason="kernel library not built")
@pytest.mark.parametrize("shape,want", FAMILY)
def test_family(shape, want):
    assert ops.lib().blitz_gemm_family(*shape) == want


# the kernel that runs where no hint is given: what is one round of 33 clusters of four, and K beyond 512, goes to those
CHOICE = [
    ((1, 4096, 4096, STORE, 1), STREAM), ((128, 4096, 4096, ADD, 1), STREAM), ((129, 4096, 4096, ADD, 1), QUAD), ((256, 6144, 4096, STORE, 1), WIDE),
    ((136, 2048, 14336, STORE, 1), STREAM), ((256, 6144, 8192, ADD, 1), PAIR), ((193, 14336, 4096, SILU, 1), WIDE), ((192, 14336, 4096, SILU, 1), STREAM),
    ((300, 2048, 4096, STORE, 1), QUAD), ((300, 2176, 4096, STORE, 1), TILED), ((300, 2048, 520, ADD, 1), QUAD), ((300, 2048, 512, ADD, 1), WIDE),
    ((300, 2048, 256, STORE, 1), WIDE), ((3000, 128, 2048, STORE, 1), QUAD), ((8448, 128, 576, STORE, 1), QUAD), ((8449, 128, 576, STORE, 1), TILED),
    ((1000, 1024, 2048, F32, 1), QUAD), ((1000, 1024, 2048, SILU, 1), WIDE), ((384, 2816, 2048, SILU, 1), TILED), ((300, 56, 4096, STORE, 1), TILED),
    ((300, 256, 192, STORE, 16), TILED), ((1574, 4096, 4096, ADD, 1), WIDE), ((300, 5632, 2048, SILU, 1), TILED),
]


@pytest.mark.skipif(not ops.available(), reason="kernel library not built")
@pytest.mark.parametrize("shape,want", CHOICE)
def test_choice(shape, want):
    assert ops.lib().blitz_gemm_choice(*shape) == want


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
        kernel = L.blitz_gemm_choice(*shape)
        assert supported[kernel](*shape), (shape, kernel)
        used.add(kernel)
    assert used == set(supported)
