"""The integer double multiply, divide and square root (nt2cuda/f64_int.cuh) against
the host's IEEE arithmetic: the header also compiles as plain C++."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HARNESS = r"""
#include "nt2cuda/f64_int.cuh"
#include <stdio.h>
#include <stdlib.h>
using namespace nt2cuda::f64i;
static uint64_t state = 88172645463325252ull;
static uint64_t rnd() { state ^= state << 7; state ^= state >> 9; return state * 0x9E3779B97F4A7C15ull; }
// significands random, or next to all zeros, all ones or one bit
static uint64_t mant()
{
  const uint64_t ones = 0xfffffffffffffull, k = rnd() % 53, small = rnd() % 8;
  uint64_t m = rnd() >> 12;
  switch (rnd() % 8) {
    case 0: m &= ~((1ull << k) - 1); break;
    case 1: m |= (1ull << k) - 1; break;
    case 2: m = small; break;
    case 3: m = ones - small; break;
    case 4: m = (1ull << k) + small - 4; break;
  }
  return m & ones;
}
static double any(int lo, int hi)
{
  const uint64_t e = rnd() % 8 ? (uint64_t)lo + rnd() % (uint64_t)(hi - lo + 1) : (rnd() & 1 ? lo : hi);
  return from_bits((rnd() & 0x8000000000000000ull) | (e << 52) | mant());
}
static bool same(double a, double b) { return bits(a) == bits(b) || (a != a && b != b); }
int main(int argc, char** argv)
{
  const int which = atoi(argv[1]);
  seed_skew() = atoi(argv[2]);
  const long n = atol(argv[3]);
  long bad = 0;
  for (long i = 0; i < n; ++i) {
    // the integer forms over their whole range, then the checked ones over every exponent
    const double a = any(512, 1534), b = any(512, 1534), p = any(513, 1534), q = any(513, 1534);
    const double u = any(0, 2047), v = any(0, 2047);
    if (which == 0) bad += !same(mul_int(a, b), a * b) + !same(mul(u, v), u * v);
    else if (which == 1) bad += !same(div_int(p, q), p / q) + !same(div(u, v), u / v);
    else {
      const double s = from_bits(bits(a) & 0x7fffffffffffffffull);
      const double t = from_bits((bits(s) & 0xffffff8000000ull) | 0x3ff0000000000000ull);   // an exact square
      bad += !same(sqrt_int(s), ::sqrt(s)) + !same(sqrt_int(t * t), t) + !same(nt2cuda::f64i::sqrt(u), ::sqrt(u));
    }
  }
  printf("%ld\n", bad);
  return 0;
}
"""


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("f64int")
    (d / "h.cpp").write_text(HARNESS)
    exe = d / "h"
    subprocess.run([gxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(ROOT, "nt2_gb300", "csrc"),
                    str(d / "h.cpp"), "-o", str(exe)], check=True)
    return str(exe)


# the quotient's and root's seeds: correctly rounded, and one unit to either side
@pytest.mark.parametrize("which,name", [(0, "multiply"), (1, "divide"), (2, "square root")])
@pytest.mark.parametrize("skew", [-1, 0, 1])
def test_integer_form_is_correctly_rounded(harness, which, name, skew):
    r = subprocess.run([harness, str(which), str(skew), "2000000"], capture_output=True, text=True, check=True)
    assert int(r.stdout) == 0, name
