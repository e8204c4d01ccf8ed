"""The largest kernel volumes that wide layers run on the tensor-core kernels with: beside the operands the tile table takes eight
bytes of shared memory per offset, so what else the kernel keeps there decides where they end (no GPU: 227 KB are assumed)."""
import pytest

from fgms_b200 import _lib


@pytest.mark.parametrize("c_in,c_out,dtype,math,k_vol", [
    (256, 256, _lib.DTYPE_F16, _lib.MATH_F16, 2786),
    (240, 208, _lib.DTYPE_F16, _lib.MATH_F16, 3810),
    (128, 256, _lib.DTYPE_F32, _lib.MATH_TF32, 2786),
    (160, 208, _lib.DTYPE_F32, _lib.MATH_TF32, 1250),
    (192, 192, _lib.DTYPE_F32, _lib.MATH_TF32, 738),
    (256, 128, _lib.DTYPE_F32, _lib.MATH_TF32, 2786),
])
def test_forward_and_input_gradient_up_to_k_vol(c_in, c_out, dtype, math, k_vol):
    family = _lib.lib.fgms_b200_kernel_family
    assert family(0, c_in, c_out, k_vol, dtype, math) == 1
    assert family(1, c_out, c_in, k_vol, dtype, math) == 1  # the same operand sizes the other way round
