"""Which kernel takes a product of 129 to 256 rows (no GPU; needs the built library)."""
import pytest

from blitz_scale_b200 import ops

STREAM, PAIR, WIDE, QUAD = 1, 2, 3, 4
STORE, ADD, SILU, F32 = 0, 1, 2, 5

# rows, columns, depth, epilogue -> kernel, as measured on both sides of the lines
CASES = [
    ((136, 4096, 4096, ADD), QUAD), ((256, 4096, 4096, ADD), QUAD), ((256, 4096, 14336, ADD), QUAD), ((136, 2048, 14336, STORE), STREAM),
    ((192, 2048, 14336, STORE), STREAM), ((136, 1024, 4096, STORE), STREAM), ((256, 1024, 4096, STORE), QUAD), ((256, 4096, 1024, ADD), QUAD),
    ((136, 2048, 2048, F32), STREAM), ((256, 2048, 2048, F32), QUAD), ((256, 2048, 64, STORE), WIDE),
    ((144, 6144, 4096, STORE), STREAM), ((256, 6144, 4096, STORE), WIDE), ((256, 6144, 8192, ADD), PAIR), ((144, 128256, 4096, STORE), STREAM),
    ((256, 128256, 4096, STORE), WIDE), ((256, 8192, 1024, STORE), WIDE),
    ((192, 14336, 4096, SILU), STREAM), ((193, 14336, 4096, SILU), WIDE), ((144, 8192, 4096, SILU), WIDE),
]


@pytest.mark.skipif(not ops.available(), reason="kernel library not built")
@pytest.mark.parametrize("shape,want", CASES)
def test_few_rows(shape, want):
    assert ops.lib().blitz_gemm_few_rows(*shape) == want
    M, N, K, epilogue = shape
    supported = {STREAM: lambda: ops.lib().blitz_gemm_decode_supported(M, N, K, 0, epilogue), PAIR: lambda: ops.lib().blitz_gemm_pair_supported(M, N, K, 0, epilogue),
                 WIDE: lambda: ops.lib().blitz_gemm_wide_supported(M, N, K, 0, epilogue, 1), QUAD: lambda: ops.lib().blitz_gemm_quad_supported(M, N, K, 0, epilogue)}
    assert supported[want]()
