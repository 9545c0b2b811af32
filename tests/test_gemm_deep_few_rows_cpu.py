"""Which kernel takes a deep product of 129 to 256 rows that is too wide for one round of clusters (no GPU; needs the built library)."""
import pytest

from blitz_scale_b200 import ops

STREAM, PAIR, WIDE = 1, 2, 3
STORE, ADD = 0, 1

# rows, columns, depth, epilogue -> the fastest as measured, by 5 % and more
CASES = [
    ((192, 6144, 8192, ADD), PAIR), ((224, 6144, 8192, ADD), PAIR), ((136, 6144, 8192, STORE), STREAM), ((224, 6144, 14336, STORE), PAIR),
    ((256, 5120, 8192, ADD), PAIR), ((136, 5120, 8192, ADD), STREAM), ((256, 5632, 14336, ADD), PAIR), ((208, 5632, 14336, STORE), PAIR),
    ((192, 8192, 14336, STORE), STREAM), ((160, 8192, 8192, STORE), STREAM), ((256, 8192, 14336, STORE), PAIR), ((208, 9216, 11008, ADD), PAIR),
    ((240, 4352, 14336, STORE), PAIR), ((176, 4352, 14336, STORE), STREAM), ((224, 7168, 11008, ADD), PAIR), ((160, 7168, 11008, ADD), STREAM),
]


@pytest.mark.skipif(not ops.available(), reason="kernel library not built")
@pytest.mark.parametrize("shape,want", CASES)
def test_deep_few_rows(shape, want):
    assert ops.lib().blitz_gemm_few_rows(*shape) == want
