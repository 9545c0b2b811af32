"""What the rule for products takes a device to hold: asked of the device; the same choices as without one (tests/test_gemm_kernel_cpu.py) where the answers are the same."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_resident():
    from blitz_scale_b200 import ops
    got = [ops.lib().blitz_gemm_resident(i) for i in range(10)]
    assert got[0] == got[1] == torch.cuda.get_device_properties(0).multi_processor_count
    assert all(0 < got[i] * i <= got[0] for i in range(1, 9)) and 0 < 4 * got[9] <= got[0]
    print(got)
    if got == [148, 148, 74, 45, 33, 26, 22, 15, 15, 33]:       # (how many clusters fit depends on which SMs of a chip are in use)
        from test_gemm_kernel_cpu import KERNEL
        assert all(ops.lib().blitz_gemm_kernel(*shape) == want for shape, want in KERNEL)
