"""Which kernel takes a product: the rule that the library decides by (no GPU; needs the built library)."""
import pytest

from blitz_scale_b200 import ops

TILED, STREAM, PAIR, WIDE = 0, 1, 2, 3
STORE, ADD, SILU, F32 = 0, 1, 2, 5

# rows, columns, depth, epilogue, blocks -> kernel, as measured on both sides of every line
CASES = [
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
@pytest.mark.parametrize("shape,want", CASES)
def test_choice(shape, want):
    assert ops.lib().blitz_gemm_choice(*shape) == want
