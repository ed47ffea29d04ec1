// nt2cuda/f64_int.cuh -- correctly rounded double multiply, divide and square
// root on the 32-bit integer pipes.
//
// GB300 executes 2 double-precision operations per clock and SM (measured 1.9
// to 2.05 for add, multiply, fma, compare, rint and the conversions alike; 0.24
// divisions and 0.23 roots), against 64 to 128 integer ones, so one double
// instruction holds its pipe as long as 32 to 64 integer instructions take.  In
// dependent chains the multiply below reaches 2.6 per clock and SM, the
// division 1.1 and the root 1.1, and they run beside the additions, which stay
// on the double pipe: multiply and add together 1.85 per clock against 0.95
// for the two instructions.  2^24 exact Black-Scholes options in double take
// 2.93 ms (12.35 with the double instructions; 6.47 with these forms in the
// functors as they were written for those), sin over 3000001 doubles 79 us (256,
// 159).
//
// Results are the IEEE round-to-nearest-even ones, bit for bit.  The integer
// form covers operands whose exponents keep every intermediate normal; the
// rest (zeros, subnormals, infinities, NaNs, results near overflow or
// underflow) take the hardware instruction.
//
// The header also compiles as host C++ (without the hardware fallbacks being
// reached through CUDA intrinsics), which is how the CPU tests check it.
#pragma once
#include <stdint.h>
#if defined(__CUDACC__)
#include <cuda_runtime.h>
#define NT2_F64I __host__ __device__ __forceinline__
#else
#include <math.h>
#include <string.h>
#define NT2_F64I inline
#endif

namespace nt2cuda {
namespace f64i {

// --------------------------------------------------------------- words
// (through asm: the compiler turns integer tests of a double's bits that it
// recognises, for NaNs and zeros, back into compares on the double pipe)
NT2_F64I uint64_t bits(double a)
{
#if defined(__CUDA_ARCH__)
  uint64_t u;
  asm("mov.b64 %0, %1;" : "=l"(u) : "d"(a));
  return u;
#else
  uint64_t u;
  memcpy(&u, &a, 8);
  return u;
#endif
}
NT2_F64I double from_bits(uint64_t u)
{
#if defined(__CUDA_ARCH__)
  return __longlong_as_double((long long)u);
#else
  double a;
  memcpy(&a, &u, 8);
  return a;
#endif
}
NT2_F64I uint32_t hi32(uint64_t u) { return (uint32_t)(u >> 32); }
NT2_F64I uint32_t lo32(uint64_t u) { return (uint32_t)u; }
NT2_F64I uint64_t pack(uint32_t lo, uint32_t hi) { return ((uint64_t)hi << 32) | lo; }
// upper word of (hi:lo) << s, and lower word of (hi:lo) >> s, 0 <= s < 32
NT2_F64I uint32_t shl_hi(uint32_t lo, uint32_t hi, uint32_t s)
{
#if defined(__CUDA_ARCH__)
  return __funnelshift_l(lo, hi, s);
#else
  return hi32(pack(lo, hi) << s);
#endif
}
NT2_F64I uint32_t shr_lo(uint32_t lo, uint32_t hi, uint32_t s)
{
#if defined(__CUDA_ARCH__)
  return __funnelshift_r(lo, hi, s);
#else
  return lo32(pack(lo, hi) >> s);
#endif
}
NT2_F64I uint32_t mulhi(uint32_t a, uint32_t b)
{
#if defined(__CUDA_ARCH__)
  return __umulhi(a, b);
#else
  return hi32((uint64_t)a * b);
#endif
}
NT2_F64I uint64_t wide(uint32_t a, uint32_t b) { return (uint64_t)a * b; }

// The hardware multiply (operands outside the integer form's range).
NT2_F64I double hw_mul(double a, double b)
{
#if defined(__CUDA_ARCH__)
  return __dmul_rn(a, b);
#else
  return a * b;
#endif
}
// Single-precision reciprocal of x in [1, 2) and reciprocal square root of x in
// [1, 4), with relative errors of at most 2^-23 and 2^-22.9 (the PTX ISA's
// bounds).  They only seed the quotient and the root below.
#if !defined(__CUDACC__)
inline int& seed_skew() { static int s = 0; return s; }   // host tests: seeds off by this many units in the last place
#endif
NT2_F64I uint32_t rcp_bits(uint32_t x)
{
#if defined(__CUDA_ARCH__)
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float(x)));
  return __float_as_uint(r);
#elif !defined(__CUDACC__)
  float f;
  memcpy(&f, &x, 4);
  f = 1.0f / f;
  memcpy(&x, &f, 4);
  return x + (uint32_t)seed_skew();
#else
  return x;
#endif
}
NT2_F64I uint32_t rsqrt_bits(uint32_t x)
{
#if defined(__CUDA_ARCH__)
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float(x)));
  return __float_as_uint(r);
#elif !defined(__CUDACC__)
  float f;
  memcpy(&f, &x, 4);
  f = (float)(1.0 / ::sqrt((double)f));
  memcpy(&x, &f, 4);
  return x + (uint32_t)seed_skew();
#else
  return x;
#endif
}

// into [1/2, 1), where the bits below the exponent are the seed's significand
NT2_F64I uint32_t seed_clamp(uint32_t r)
{
  r = r < 0x3f7fffffu ? r : 0x3f7fffffu;
  return r > 0x3f000000u ? r : 0x3f000000u;
}

// Exponent fields from 512 (513) to 1534: products (quotients) of two such
// numbers are normal.
NT2_F64I bool mul_range(uint32_t h) { return (h & 0x7ff00000u) - 0x20000000u < 0x3ff00000u; }
NT2_F64I bool div_range(uint32_t h) { return (h & 0x7ff00000u) - 0x20100000u < 0x3fe00000u; }

// (hi:lo) + carry of x + y
NT2_F64I uint64_t add_carry_of(uint32_t x, uint32_t y, uint32_t lo, uint32_t hi)
{
#if defined(__CUDA_ARCH__)
  asm("{\n\t.reg .u32 t;\n\tadd.cc.u32 t, %2, %3;\n\taddc.cc.u32 %0, %0, 0;\n\taddc.u32 %1, %1, 0;\n\t}"
      : "+r"(lo), "+r"(hi)
      : "r"(x), "r"(y));
  return pack(lo, hi);
#else
  return pack(lo, hi) + hi32((uint64_t)x + y);
#endif
}

// ------------------------------------------------------------ multiply
// The 106-bit product of the 53-bit significands from four 32x32 products,
// its leading bit at 104 or 105; shifted so that it stands at bit 52 of
// (r1:r0) with the bits below in `rest`, of which the top word and whether
// anything is left decide the rounding to nearest even.  Signs and
// exponents add up in the high word: the exponents' sum less the bias fits its
// 11 bits, so the sign bits add without a carry into or out of them.
NT2_F64I double mul_int(double a, double b)
{
  const uint64_t ua = bits(a), ub = bits(b);
  const uint32_t ah = hi32(ua), al = lo32(ua), bh = hi32(ub), bl = lo32(ub);
  const uint32_t xh = (ah & 0xfffffu) | 0x100000u, yh = (bh & 0xfffffu) | 0x100000u;
  const uint64_t p0 = wide(al, bl);
  const uint64_t mid = wide(al, yh) + (wide(xh, bl) + hi32(p0));
  const uint64_t top = wide(xh, yh) + hi32(mid);
  const uint32_t th = hi32(top), d = th >> 9;                      // product >= 2
  const uint32_t s = 12u - d;
  const uint32_t r1 = shl_hi(lo32(top), th, s), r0 = shl_hi(lo32(mid), lo32(top), s);
  const uint32_t rest = shl_hi(lo32(p0), lo32(mid), s);
  // past the half, or on it with r0 odd or bits of p0 left (those of them that
  // were shifted into `rest` keep it off the half either way)
  const uint32_t below = 0x7fffffffu + ((r0 & 1u) | (lo32(p0) < 1u ? lo32(p0) : 1u));
  const uint32_t e = (ah & 0xfff00000u) + (bh & 0xfff00000u) - 0x40000000u;   // (1023 + 1) << 20: r1 holds the leading one
  return from_bits(add_carry_of(rest, below, r0, r1 + e + (d << 20)));
}
NT2_F64I double mul(double a, double b)
{
  const uint32_t ah = hi32(bits(a)), bh = hi32(bits(b));
  if (mul_range(ah) && mul_range(bh)) return mul_int(a, b);
  return hw_mul(a, b);
}
#if defined(__CUDACC__)
static __device__ __noinline__ double mul_any(double a, double b) { return mul(a, b); }   // for rarely run code
#endif

// -------------------------------------------------------------- divide
// With significands A and B, A doubled if A < B, so that q = A/B is in [1, 2),
// and b = B/2^52:
//   r1  2^32/b less at most 3: the seed R0 and one Newton step (the truncated b
//       makes it at most 2 too large before the 2 taken off);
//   q1  q 2^30 less at most 5, from r1 times the top 32 bits of A;
//   q2  floor(2^23 rem1/B) or one less, rem1 = A 2^30 - q1 B < 5 B, the same way;
// and rem2 = rem1 2^23 - q2 B says which, so that Q = q1 2^23 + q2 =
// floor(q 2^53) exactly.  A quotient of 53-bit numbers never lies half way
// between two of them, so (Q + 1) >> 1 is q rounded to nearest.
NT2_F64I double div_int(double a, double b)
{
  const uint64_t ua = bits(a), ub = bits(b);
  const uint32_t ah = hi32(ua), bh = hi32(ub), bl = lo32(ub);
  const uint32_t yh = (bh & 0xfffffu) | 0x100000u;
  const uint64_t A0 = pack(lo32(ua), (ah & 0xfffffu) | 0x100000u), B = pack(bl, yh);
  uint32_t r = rcp_bits((shl_hi(bl, bh, 3) & 0x7fffffu) | 0x3f800000u);
  r = seed_clamp(r);
  const uint32_t R0 = (r & 0x7fffffu) | 0x800000u;                 // 2^24/b
  const uint64_t P = wide(R0, shl_hi(bl, yh, 11));                 // R0 b 2^31
  const int32_t err = -(int32_t)shr_lo(lo32(P), hi32(P), 2);       // (1 - R0 b 2^-24) 2^53, below 1.5 2^30
  const uint32_t r1 = (R0 << 8) + (uint32_t)(int32_t)(((int64_t)(int32_t)(R0 << 7) * err) >> 52) - 2u;
  const uint32_t d = A0 < B ? 1u : 0u;
  const uint64_t A = A0 << d;
  const uint32_t q1 = mulhi((uint32_t)(A >> 22), r1);
  const uint64_t rem1 = (A << 30) - (uint64_t)q1 * B;              // in [0, 5 B); the products wrap, it does not
  uint32_t q2 = mulhi((uint32_t)(rem1 >> 24), r1) >> 5;
  const uint64_t rem2 = (rem1 << 23) - (uint64_t)q2 * B;           // in [0, 2 B)
  q2 += rem2 >= B ? 2u : 1u;                                       // the one missing, and 1 to round
  const uint64_t m = (((uint64_t)q1 << 23) + q2) >> 1;
  const uint32_t e = (ah & 0xfff00000u) - (bh & 0xfff00000u) + 0x3fe00000u - (d << 20);   // m holds the leading one
  return from_bits(m + pack(0u, e));
}
// Out of line: a functor has several, each some 55 instructions, and the
// statements' loop bodies already exceed the instruction cache's first levels
// (exact Black-Scholes 3.13 ms with every division inlined, 2.89 called).
#if defined(__CUDACC__)
static __device__ __noinline__ double div_mid(double a, double b) { return div_int(a, b); }
static __device__ __noinline__ double div_any(double a, double b)
{
  return div_range(hi32(bits(a))) && div_range(hi32(bits(b))) ? div_int(a, b) : __ddiv_rn(a, b);
}
#endif
NT2_F64I double div(double a, double b)
{
#if defined(__CUDA_ARCH__)
  return div_any(a, b);
#else
  return div_range(hi32(bits(a))) && div_range(hi32(bits(b))) ? div_int(a, b) : a / b;
#endif
}

// --------------------------------------------------------- square root
// a = A 2^-52 4^k with A 2^-52 =: f in [1, 4):
//   y1  2^32/sqrt(f) less at most 7: the seed Y0 and one Newton step;
//   s1  sqrt(f) 2^30 less at most 9;
//   s2  2^23 rem1/(2 sqrt(f) 2^30), rem1 = A 2^8 - s1^2, at most 2 short of
//       what is missing;
// Q = s1 2^23 + s2 is floor(sqrt(f) 2^53) or one less, and A 2^54 - Q^2 (which
// fits 64 bits though its terms wrap) says which.  A root of a 53-bit number
// never lies half way between two of them, so (Q + 1) >> 1 rounds to nearest.
NT2_F64I double sqrt_int(double a)
{
  const uint64_t ua = bits(a);
  const uint32_t ah = hi32(ua), al = lo32(ua);
  const uint32_t odd = ((ah >> 20) & 1u) ^ 1u;
  const uint64_t A = pack(al, (ah & 0xfffffu) | 0x100000u) << odd;
  uint32_t r = rsqrt_bits(((shl_hi(al, ah, 3) & 0x7fffffu) | 0x3f800000u) + (odd << 23));
  r = seed_clamp(r);
  const uint32_t Y0 = (r & 0x7fffffu) | 0x800000u;                  // 2^24/sqrt(f)
  const uint32_t a32 = (uint32_t)(A >> 22);                         // f 2^30
  const uint32_t g = (uint32_t)(wide(a32, Y0) >> 24);               // sqrt(f) 2^30
  const uint64_t G = wide(g, Y0);                                   // f Y0^2 2^-48 2^54
  const int32_t err = -(int32_t)shr_lo(lo32(G), hi32(G), 2);        // (1 - f Y0^2 2^-48) 2^52, below 2^31
  const uint32_t y1 = (Y0 << 8) + (uint32_t)(int32_t)(((int64_t)(int32_t)(Y0 << 7) * err) >> 52) - 5u;
  const uint32_t s1 = mulhi(a32, y1);
  const uint64_t rem1 = (A << 8) - wide(s1, s1);                    // below 2^35
  const uint32_t s2 = mulhi((uint32_t)(rem1 >> 3), y1) >> 5;
  uint64_t Q = ((uint64_t)s1 << 23) + s2;
  const uint64_t rem2 = (A << 54) - Q * Q;                          // (T - Q)(T + Q), T = sqrt(f) 2^53
  Q += rem2 > 2u * Q ? 2u : 1u;
  const uint32_t e = ((ah >> 20) - odd + 1021u) >> 1;               // Q >> 1 holds the leading one
  return from_bits((Q >> 1) + pack(0u, e << 20));
}
// positive, exponent field 512 to 1534
NT2_F64I bool sqrt_range(uint32_t h) { return h - 0x20000000u < 0x3ff00000u; }
#if defined(__CUDACC__)
static __device__ __noinline__ double sqrt_any(double a) { return sqrt_range(hi32(bits(a))) ? sqrt_int(a) : __dsqrt_rn(a); }
#endif
NT2_F64I double sqrt(double a)
{
#if defined(__CUDA_ARCH__)
  return sqrt_any(a);
#else
  return sqrt_range(hi32(bits(a))) ? sqrt_int(a) : ::sqrt(a);
#endif
}

// ------------------------------------------------- small conversions
// (double)k for |k| < 2^22: the float of k (exact) with its exponent rebiased.
NT2_F64I double small_int(int k)
{
#if defined(__CUDA_ARCH__)
  const uint32_t f = __float_as_uint(__int_as_float(0x4b400000 + k) - 12582912.0f);
#else
  const float v = (float)k;
  uint32_t f;
  memcpy(&f, &v, 4);
#endif
  const uint32_t h = ((uint32_t)((int32_t)f >> 3) & 0x8fffffffu) + 0x38000000u;
  return from_bits(pack(f << 29, k ? h : 0u));
}
// rint(t) as an integer and as a double, for |t| < 2^22 (unspecified beyond):
// one addition on the double pipe, where rint and the conversion take two.
NT2_F64I double round_small(double t, int& k)
{
#if defined(__CUDA_ARCH__)
  k = (int)lo32(bits(__dadd_rn(t, 6755399441055744.0)));
#else
  k = (int)lo32(bits(t + 6755399441055744.0));
#endif
  return small_int(k);
}
// k*c for k = small_int(n), c a normal constant of moderate size (k = 0 is no operand of the integer multiply)
NT2_F64I double mul_small(double k, int n, double c) { return n ? mul_int(k, c) : 0.0; }
// x * 2^n where the caller knows x and the result to be normal
NT2_F64I double scale(double x, int n) { return from_bits(bits(x) + pack(0u, (uint32_t)n << 20)); }
// x / 2
NT2_F64I double half(double x)
{
  if ((hi32(bits(x)) & 0x7fffffffu) - 0x00200000u < 0x7fd00000u) return scale(x, -1);
  return hw_mul(x, 0.5);
}
// x < c for x >= 0 or NaN without its sign, c > 0: the bits compare as integers
NT2_F64I bool below(double x, double c) { return bits(x) < bits(c); }
// an integer that orders doubles (not NaNs) as < does; both zeros are 0
NT2_F64I int64_t order_key(double x)
{
  const int64_t m = (int64_t)(bits(x) & 0x7fffffffffffffffull);
  return (int32_t)hi32(bits(x)) < 0 ? -m : m;
}
// the high word without its sign: |x| >= 2^e and non-finite tests on the top 32 bits
NT2_F64I uint32_t abs_hi(double x) { return hi32(bits(x)) & 0x7fffffffu; }
NT2_F64I bool is_zero(double x) { return (bits(x) << 1) == 0ull; }

// --------------------------------------------------- fixed point frames
// A block of doubles as 64-bit integers in units of 2^(F - 1075 - SH), F at
// least every element's biased exponent: an element's significand, SH bits up,
// shifted down by what its exponent lacks (elements more than SH bits below F
// lose their lowest bits; zeros and far smaller ones become 0).
NT2_F64I uint64_t shr64(uint64_t v, uint32_t n)     // 0 for n >= 64
{
#if defined(__CUDA_ARCH__)
  uint64_t r;
  asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(n));
  return r;
#else
  return n > 63u ? 0ull : v >> n;
#endif
}
template <int SH> NT2_F64I int64_t to_fixed(double x, uint32_t F)
{
  const uint64_t u = bits(x);
  const uint32_t h = hi32(u);
  const uint64_t m = pack(lo32(u), (h & 0xfffffu) | 0x100000u) << SH;
  const int64_t v = (int64_t)shr64(m, F - ((h >> 20) & 0x7ffu));
  return (int32_t)h < 0 ? -v : v;
}
// largest biased exponent of a block
template <int N> NT2_F64I uint32_t max_exponent(const double (&x)[N])
{
  uint32_t m = 0u;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const uint32_t h = abs_hi(x[i]);
    m = h > m ? h : m;
  }
  return m >> 20;
}
}  // namespace f64i
}  // namespace nt2cuda
