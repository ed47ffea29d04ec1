"""The double functors' multiply, divide and square root run on the integer pipes
(nt2cuda/f64_int.cuh); on the GPU they give the hardware instructions' bits over
2^30 drawn operand pairs each, every exponent and the integer forms' range ends among them."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("which,name", [(0, "multiply"), (1, "divide"), (2, "square root")])
def test_integer_form_gives_the_hardware_bits(gpu, cuda_lib, which, name):
    n = C.c_ulonglong(99)
    st = cuda_lib.nt2cuda_selftest_f64(C.c_int(which), C.byref(n), C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert st == 0
    assert n.value == 0, name
