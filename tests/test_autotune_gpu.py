"""The tuner times what a kernel has: the double Black-Scholes kernel has one unroll, so a tuned
table names no other."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", ["bs_f64", "bs_f64_fused"])
@pytest.mark.parametrize("n", [1000, 4096, 20000, 65536])
def test_double_black_scholes_has_one_unroll(gpu, cuda_lib, kernel, n):
    u, w, ms = gpu.autotune(kernel, n)
    assert u == 1 and w in (1, 2, 4, 8) and ms > 0
