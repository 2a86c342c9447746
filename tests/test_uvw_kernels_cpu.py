"""Which forward kernel a shared-weight FP32 'uvw' product takes: both tensor-core kernels have 21 warps, the one with the weights in
tensor memory (uvw_ts_kernels.cuh) four operand stages and the one with them in shared memory (uvw_tc_kernels.cuh) two."""
import pytest

import openequivariance_b200 as oeq
from openequivariance_b200 import _native

TENSOR, SHARED = 4, 2


def stages(*irreps):
    info = _native.TPHandle(oeq.FullyConnectedTPProblem(*irreps)).launch_info(0)
    assert info["threads"] == 21 * 32
    return info["stages"]


@pytest.mark.parametrize("irreps,kernel", [
    (("64x1o+64x2e", "0e+1o", "64x1o"), TENSOR),
    (("64x1o+66x2e", "0e+1o", "64x1o"), SHARED),            # rows of X in no whole pieces of four channels
    (("64x1o+64x2e", "0e+1o", "80x1o"), SHARED),            # more than 64 output channels
    (("32x0e", "0e", "32x0e"), SHARED),                     # too few slices of input channels
    (("64x1o", "0e", "64x1o"), SHARED),
    (("96x1o", "0e", "64x1o"), TENSOR),
    (("64x2e", "0e", "64x2e"), TENSOR),
])
def test_kernel_with_the_weights_in_tensor_memory(irreps, kernel):
    assert stages(*irreps) == kernel
