// nt2cuda/fold.cuh -- inner_fold (contiguous) and outer_fold (strided)
// reductions of an elementwise expression.
//
// NT2 maps sum/globalsum to inner_fold when the reduced dimension is the
// first non-singleton one and to outer_fold otherwise
// (modules/core/reduction/include/nt2/dsl/functions/reduction/run.hpp:30-104).
//   inner_fold: per outer slice, an N-lane accumulation over contiguous
//     elements, a horizontal sum and a scalar tail
//     (modules/core/reduction/include/nt2/core/functions/simd/inner_fold.hpp:49-66);
//     the OpenMP spawner splits long slices into blocks whose partials are
//     combined in arrival order (modules/arch/openmp/include/nt2/sdk/openmp/spawner/fold.hpp:49-66).
//   outer_fold: out[o][i] = fold over m of in[o][m][i], contiguous in i
//     (modules/core/reduction/include/nt2/core/functions/details/outer_fold_step.hpp:33-67).
// Here the element values come from an expression (so globalsum(X*Y) reads X
// and Y once, as NT2's fused fold_step does), FP32 accumulates with
// TwoSum-compensated partials when COMP is set, and the split of the work
// into warps and blocks depends only on the table's shape (and on whether the
// call is captured into a graph, captured_cut): partials are combined in index
// order, never in arrival order, so results are bitwise reproducible from run to
// run and across GPUs.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include "expr.cuh"
#include "math.cuh"

namespace nt2cuda {
namespace fold {

// ------------------------------------------------ compensated accumulators
template <class T> struct acc { T s, c; };

template <bool COMP, class T> __device__ __forceinline__ void add(acc<T>& a, T x)
{
  using namespace math;
  if constexpr (COMP) {
    T t = nt2cuda::math::add(a.s, x);
    T z = sub(t, a.s);
    T e = nt2cuda::math::add(sub(a.s, sub(t, z)), sub(x, z));
    a.c = nt2cuda::math::add(a.c, e);
    a.s = t;
  } else {
    a.s = nt2cuda::math::add(a.s, x);
  }
}

template <bool COMP, class T> __device__ __forceinline__ acc<T> merge(acc<T> a, acc<T> b)
{
  using namespace math;
  if constexpr (COMP) {
    T t = nt2cuda::math::add(a.s, b.s);
    T z = sub(t, a.s);
    T e = nt2cuda::math::add(sub(a.s, sub(t, z)), sub(b.s, z));
    return acc<T>{t, nt2cuda::math::add(nt2cuda::math::add(a.c, b.c), e)};
  } else {
    return acc<T>{nt2cuda::math::add(a.s, b.s), T(0)};
  }
}

// The value of a compensated pair.  Once the running sum is not finite (an
// overflow, an infinite or NaN term) its compensation is NaN and the sum
// itself is the result, as in NT2's plain float sum: inf stays inf.
template <bool COMP, class T> __device__ __forceinline__ T result(acc<T> a)
{
  if constexpr (COMP) {
    const T r = nt2cuda::math::add(a.s, a.c);
    return r != r ? a.s : r;
  } else {
    return a.s;
  }
}

// ------------------------------------------------------------ operations
// A reduction is NT2's reduction_<Tag, Bop, Neutral>
// (boost/simd/reduction/functions/sum.hpp:26-29, maximum.hpp:30, minimum.hpp:29,
// prod.hpp:26, all.hpp:29, any.hpp:29) applied to the elements of an expression,
// plus the scalar step that turns the fold into mean, norm2, var or stdev
// (nt2/core/functions/expr/mean.hpp, norm2.hpp, var.hpp, stdev.hpp).  An
// operation supplies its accumulator (state), the neutral state, add,
// merge (the left operand holds the lower indices), warp shuffles, uncached
// loads of partials, and finish(state, n) -> output for a fold of n elements.
enum fin_kind { FIN_NONE = 0, FIN_SQRT = 1, FIN_MEAN = 2 };

template <bool COMP, int FIN = FIN_NONE> struct op_sum {
  template <class T> using state = acc<T>;
  template <class T> using out_t = T;
  template <class T> __device__ __forceinline__ static state<T> init() { return acc<T>{T(0), T(0)}; }
  template <class T> __device__ __forceinline__ static void add(state<T>& a, T x) { fold::add<COMP>(a, x); }
  template <class T> __device__ __forceinline__ static state<T> merge(state<T> a, state<T> b) { return fold::merge<COMP>(a, b); }
  template <class T> __device__ __forceinline__ static state<T> shfl(state<T> a, int off)
  {
    return acc<T>{__shfl_xor_sync(0xffffffffu, a.s, off), __shfl_xor_sync(0xffffffffu, a.c, off)};
  }
  template <class T> __device__ __forceinline__ static state<T> ldcg(const state<T>* p)
  {
    return acc<T>{__ldcg(&p->s), __ldcg(&p->c)};
  }
  template <class T> __device__ __forceinline__ static state<T> shfl_from(state<T> a, int src)
  {
    return acc<T>{__shfl_sync(0xffffffffu, a.s, src), __shfl_sync(0xffffffffu, a.c, src)};
  }
  template <class T> __device__ __forceinline__ static T finish(state<T> a, size_t n)
  {
    const T r = result<COMP>(a);
    if constexpr (FIN == FIN_SQRT) return math::sqrt_(r);
    if constexpr (FIN == FIN_MEAN) return math::mul(math::div(T(1), (T)n), r);   // rec(n) * sum
    return r;
  }
};

template <class T> struct val { T v; };

// max / min / prod: one value; max and min ignore NaNs (NT2's result with NaNs
// depends on its evaluation order), their neutral elements are NT2's Maxinit
// (-largest finite) and Valmax (+largest finite).  KIND 3 and 4 are max and min
// with the neutral elements of cummax and cummin, Minf and Inf
// (boost/simd/swar/functions/cummax.hpp, cummin.hpp).
template <int KIND> struct op_val {   // 0 max, 1 min, 2 prod, 3 cummax, 4 cummin
  template <class T> using state = val<T>;
  template <class T> using out_t = T;
  template <class T> __device__ __forceinline__ static state<T> init()
  {
    // largest finite value: NT2's Valmax, and -Valmax is its Maxinit (constant/constants/maxinit.hpp)
    const T big = sizeof(T) == 4 ? (T)3.40282346638528859812e+38 : (T)1.79769313486231570815e+308;
    const T inf = sizeof(T) == 4 ? (T)__int_as_float(0x7f800000) : (T)__longlong_as_double(0x7ff0000000000000ll);
    if constexpr (KIND == 2) return val<T>{T(1)};
    else if constexpr (KIND == 3) return val<T>{-inf};
    else if constexpr (KIND == 4) return val<T>{inf};
    else return val<T>{KIND == 0 ? -big : big};
  }
  // a is the accumulator (never NaN), b the next element: NT2's max(a,b) = a > b ? a : b
  // (boost/simd/arithmetic/functions/scalar/max.hpp), except that a NaN b is skipped
  // For doubles the comparison is of integers (magnitude, negated where the sign
  // is set, so that the zeros are equal): two compares on the double pipe would
  // take 32 clocks a warp, three times what the memory takes.
  template <class T> __device__ __forceinline__ static T op(T a, T b)
  {
    if constexpr (sizeof(T) == 8 && KIND != 2) {
      const int64_t ka = f64i::order_key(a), kb = f64i::order_key(b);
      const bool nan = (f64i::bits(b) << 1) > 0xffe0000000000000ull;
      return ((KIND == 0 || KIND == 3) ? ka > kb : ka < kb) || nan ? a : b;
    }
    if constexpr (KIND == 0 || KIND == 3) return (a > b || b != b) ? a : b;
    else if constexpr (KIND == 1 || KIND == 4) return (a < b || b != b) ? a : b;
    else return math::mul(a, b);
  }
  template <class T> __device__ __forceinline__ static void add(state<T>& a, T x) { a.v = op(a.v, x); }
  template <class T> __device__ __forceinline__ static state<T> merge(state<T> a, state<T> b) { return val<T>{op(a.v, b.v)}; }
  template <class T> __device__ __forceinline__ static state<T> shfl(state<T> a, int off)
  {
    return val<T>{__shfl_xor_sync(0xffffffffu, a.v, off)};
  }
  template <class T> __device__ __forceinline__ static state<T> ldcg(const state<T>* p) { return val<T>{__ldcg(&p->v)}; }
  template <class T> __device__ __forceinline__ static state<T> shfl_from(state<T> a, int src)
  {
    return val<T>{__shfl_sync(0xffffffffu, a.v, src)};
  }
  template <class T> __device__ __forceinline__ static T finish(state<T> a, size_t) { return a.v; }
};

// all / any: logical_and / logical_or of (x != 0) with neutral True / False;
// none = !any (boost/simd/reduction/functions/scalar/none.hpp: is_eqz of the
// element).  The output is a logical table stored as uint8_t 0/1.
template <bool ANY, bool NOT = false> struct op_logic {
  using flag = val<unsigned>;
  template <class T> using state = flag;
  template <class T> using out_t = uint8_t;
  template <class T> __device__ __forceinline__ static flag init() { return flag{ANY ? 0u : 1u}; }
  template <class T> __device__ __forceinline__ static void add(flag& a, T x)
  {
    const unsigned b = (x != T(0)) ? 1u : 0u;
    a.v = ANY ? (a.v | b) : (a.v & b);
  }
  __device__ __forceinline__ static flag merge(flag a, flag b) { return flag{ANY ? (a.v | b.v) : (a.v & b.v)}; }
  __device__ __forceinline__ static flag shfl(flag a, int off) { return flag{__shfl_xor_sync(0xffffffffu, a.v, off)}; }
  __device__ __forceinline__ static flag ldcg(const flag* p) { return flag{__ldcg(&p->v)}; }
  __device__ __forceinline__ static uint8_t finish(flag a, size_t) { return (uint8_t)(NOT ? (a.v ^ 1u) : a.v); }
};

// var / stdev in one pass: Welford's update per element and Chan's merge of
// partial (count, mean, M2).  NT2 computes var(A) = f * asum2(center(A)) with
// f = rec(n - 1) (rec(n) with w = 1, 1 when n <= 1) in two passes
// (nt2/core/functions/expr/var.hpp); the result here is the same quantity
// within the error bound stated in the tests.
template <class T> struct moments { T n, mean, m2; };

template <bool W1, bool STDEV> struct op_moments {
  template <class U> using state = moments<U>;
  template <class U> using out_t = U;
  template <class U> __device__ __forceinline__ static state<U> init() { return moments<U>{U(0), U(0), U(0)}; }
  template <class U> __device__ __forceinline__ static void add(state<U>& a, U x)
  {
    a.n = a.n + U(1);
    const U d = x - a.mean;
    if constexpr (sizeof(U) == 4) a.mean = __fmaf_rn(d, __frcp_rn(a.n), a.mean);
    else a.mean = a.mean + math::div(d, a.n);
    a.m2 = a.m2 + d * (x - a.mean);
  }
  template <class U> __device__ __forceinline__ static state<U> merge(state<U> a, state<U> b)
  {
    if constexpr (sizeof(U) == 8) {
      // five operations on the double pipe (2 a clock and SM): the counts are
      // tested as integers, the division and products are the integer ones
      if (f64i::is_zero(b.n)) return a;
      if (f64i::is_zero(a.n)) return b;
      const U n = a.n + b.n;
      const U d = b.mean - a.mean;
      const U wb = math::div(b.n, n);
      return moments<U>{n, __fma_rn(d, wb, a.mean), __fma_rn(math::mul(math::mul(d, d), a.n), wb, a.m2 + b.m2)};
    } else {
      if (b.n == U(0)) return a;
      if (a.n == U(0)) return b;
      const U n = a.n + b.n;
      const U d = b.mean - a.mean;
      const U wb = b.n / n;
      return moments<U>{n, a.mean + d * wb, a.m2 + b.m2 + d * d * a.n * wb};
    }
  }
  // N values at once (N a power of two): the block's own mean and sum of
  // squared deviations in two passes over registers, then one merge, so the
  // division of Welford's update is paid once per block instead of per value.
  template <class U, int N> __device__ __forceinline__ static void add_block(state<U>& a, const U (&x)[N])
  {
    static_assert((N & (N - 1)) == 0, "add_block: N a power of two");
    U s = x[0];
#pragma unroll
    for (int i = 1; i < N; ++i) s = s + x[i];
    const U mb = s * (U(1) / U(N));               // exact scaling
    U m2 = U(0);
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const U d = x[i] - mb;
      m2 = m2 + d * d;
    }
    a = merge(a, moments<U>{U(N), mb, m2});
  }
  template <class U> __device__ __forceinline__ static state<U> shfl(state<U> a, int off)
  {
    return moments<U>{__shfl_xor_sync(0xffffffffu, a.n, off), __shfl_xor_sync(0xffffffffu, a.mean, off),
                      __shfl_xor_sync(0xffffffffu, a.m2, off)};
  }
  template <class U> __device__ __forceinline__ static state<U> ldcg(const state<U>* p)
  {
    return moments<U>{__ldcg(&p->n), __ldcg(&p->mean), __ldcg(&p->m2)};
  }
  template <class U> __device__ __forceinline__ static U finish(state<U> a, size_t n)
  {
    const U n1 = (U)n - (W1 ? U(0) : U(1));
    const U f = (n <= 1) ? U(1) : math::div(U(1), n1);
    const U v = math::mul(f, a.m2);
    return STDEV ? math::sqrt_(v) : v;
  }
};

template <class Op, class T> using state_of = typename Op::template state<T>;

// Operations that take the values of one load trip as a block, through a
// lane-local accumulator: add(state, values) and, at the end, flush(state).
template <class Op, class T, class E> struct block_acc { static constexpr bool value = false; };

// var / stdev of floats: one Chan merge per block (op_moments::add_block).
template <bool W1, bool SD, class E> struct block_acc<op_moments<W1, SD>, float, E> {
  static constexpr bool value = true;
  using S = moments<float>;
  template <int N> __device__ __forceinline__ void add(S& a, const float (&x)[N]) { op_moments<W1, SD>::add_block(a, x); }
  __device__ __forceinline__ void flush(S&) {}
};

// Plain sums of doubles read straight from a table: a lane keeps the sum of up to
// 1024 values as an exact 96-bit integer in one fixed point frame, two bits above
// its first block's largest exponent.  A block with a value above the frame, or one
// that would lose bits in it, is added to the sum in double, value by value.  So no
// bit of a value is dropped, and the sum is rounded twice a frame where additions
// one by one round at each.  An addition holds GB300's double pipe 16 clocks a
// warp, more than the 11 in which the memory delivers the warp's 256 bytes; the
// integer form takes about 8.  4096 x 4096: columns 41.5 us one by one, 23.2 in
// frames, rows 40.4 and 26.5; with a zero in every block (or 30 binary orders)
// 47 and 49.
template <class E> struct plain_term { static constexpr bool value = false; };
template <class T> struct plain_term<term<T>> { static constexpr bool value = true; };
template <class T> struct plain_term<node<tag::abs_, term<T>>> { static constexpr bool value = true; };
template <int FIN, class E> struct block_acc<op_sum<false, FIN>, double, E> {
  static constexpr bool value = plain_term<E>::value;
  using S = acc<double>;
  static constexpr int MOST = 1024;        // values in a frame: each below 2^21 in w2
  uint32_t F = 0u;                         // the frame's exponent; 0: none
  int n = 0;                               // values in it
  uint32_t w0 = 0u, w1 = 0u, w2 = 0u;      // their sum, in units of 2^(F - 1107)

  template <int N> __device__ __forceinline__ void add(S& a, const double (&x)[N])
  {
    static_assert(N <= 16, "block of at most 16 values");
    if (F == 0u) F = frame(f64i::max_exponent(x));
    if (__builtin_expect(F != 0u && n <= MOST - N && trip(x), 1)) return;
#pragma unroll
    for (int i = 0; i < N; ++i) a.s = math::add(a.s, x[i]);
    if (n > MOST - N || f64i::max_exponent(x) > F) {    // the next block opens another
      flush(a);
      F = 0u;
    }
  }
  // for a block whose largest exponent is f; none for infinities, NaNs and the largest values
  __device__ __forceinline__ static uint32_t frame(uint32_t f) { return f < 2000u ? (f > 128u ? f : 128u) + 2u : 0u; }
  // The values into the open frame; false (and nothing added) if one is above it or
  // more than 31 bits below.  (F is at least 130, so that no exponent above it is
  // within 31 below modulo 2^11.)  Two passes over the values, so that the sums of
  // the second go to the frame itself.
  template <int N> __device__ __forceinline__ bool trip(const double (&x)[N])
  {
    uint32_t top = F << 21 | 0x1fffffu, out = 0u;      // top - 2h is the shift, 21 bits up
#pragma unroll
    for (int i = 0; i < N; ++i) out |= top - 2u * f64i::hi32(f64i::bits(x[i]));
    if (out >> 26) return false;
    asm("" : "+r"(top));                                // (computed again, not kept)
    uint32_t minus = 0u;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const uint64_t u = f64i::bits(x[i]);
      const uint32_t h = f64i::hi32(u), l = f64i::lo32(u), sh = (top - 2u * h) >> 21, m = (h & 0xfffffu) | 0x100000u;
      const uint32_t sg = (uint32_t)((int32_t)h >> 31);
      minus -= sg;                                      // -v = ~v + 1
      add96(w0, w1, w2, f64i::shr_lo(0u, l, sh) ^ sg, f64i::shr_lo(l, m, sh) ^ sg, (m >> sh) ^ sg);
    }
    add96(w0, w1, w2, minus, 0u, 0u);
    n += N;
    return true;
  }
  __device__ __forceinline__ static void add96(uint32_t& a0, uint32_t& a1, uint32_t& a2, uint32_t b0, uint32_t b1, uint32_t b2)
  {
    asm("add.cc.u32 %0, %0, %3;\n\taddc.cc.u32 %1, %1, %4;\n\taddc.u32 %2, %2, %5;"
        : "+r"(a0), "+r"(a1), "+r"(a2)
        : "r"(b0), "r"(b1), "r"(b2));
  }
  // a.s + the frame's sum, which is rounded once: its leading 64 bits (or all 96,
  // if the upper 32 are 0), those below them as one sticky bit
  __device__ __forceinline__ void flush(S& a)
  {
    if (n == 0) return;
    const uint32_t sg = (uint32_t)((int32_t)w2 >> 31);
    w0 ^= sg;
    w1 ^= sg;
    w2 ^= sg;
    add96(w0, w1, w2, sg & 1u, 0u, 0u);
    const int z = min(__clzll((long long)f64i::pack(w1, w2)), 32);
    const uint32_t low = z < 32 ? w0 << z : 0u;
    const uint64_t t = (f64i::pack(w1, w2) << z) | (z ? w0 >> (32 - z) : 0u) | (low ? 1u : 0u);
    const uint64_t v = f64i::bits(__ull2double_rn(t)) + f64i::pack(0u, (F - 1075u - (uint32_t)z) << 20);
    if (t != 0ull) a.s = math::add(a.s, f64i::from_bits(v | f64i::pack(0u, sg & 0x80000000u)));
    n = 0;
    w0 = w1 = w2 = 0u;
  }
};

// Count, mean and M2 of n values in a fixed point frame of unit 2^(F - 1075 - SH),
// from a pivot P and the exact sums s of d = value - P (128 bits) and q of d^2 (192):
// M2 = q - s^2/n.  The pivot is a few values' mean, and q may be far above M2 (n/N
// times, for the mean of N values that the rest are far from); where M2 is less than
// a quarter of q, frame_recentred moves the sums first.
template <int SH>
__device__ __forceinline__ moments<double> frame_result(double cnt, uint32_t F, int64_t P, double md, double m2)
{
  const double unit = f64i::from_bits((uint64_t)(F - 1075u - (uint32_t)SH + 1023u) << 52);
  return moments<double>{cnt, ((double)P + md) * unit, fmax(m2, 0.0) * unit * unit};
}
constexpr double kTwo64 = 18446744073709551616.0;
// To c, the mean of d rounded to a whole unit or nearly, while the sums are integers:
// s - n c and q - c (s + (s - n c)).  What is left cancels nothing.
template <int SH>
__device__ __forceinline__ moments<double> frame_recentred(int n, uint32_t F, int64_t P, int64_t s_hi, uint64_t s_lo, uint64_t q_x,
                                                        uint64_t q_hi, uint64_t q_lo)
{
  const double cnt = (double)n;
  const int64_t c = __double2ll_rn(math::div(__fma_rn((double)s_hi, kTwo64, (double)s_lo), cnt));
  const int64_t r = (int64_t)(s_lo - (uint64_t)n * (uint64_t)c);         // s - n c, 2^8 n at most
  uint64_t v_lo = s_lo + (uint64_t)r;
  uint64_t v_hi = (uint64_t)(s_hi + (r >> 63) + (v_lo < s_lo ? 1 : 0));
  const bool vn = (int64_t)v_hi < 0, cn = c < 0;
  if (vn) {
    v_hi = ~v_hi + (v_lo == 0ull ? 1ull : 0ull);
    v_lo = 0ull - v_lo;
  }
  const uint64_t u = cn ? 0ull - (uint64_t)c : (uint64_t)c;
  const unsigned __int128 p0 = (unsigned __int128)u * v_lo, p1 = (unsigned __int128)u * v_hi + (uint64_t)(p0 >> 64);
  uint64_t w0 = (uint64_t)p0, w1 = (uint64_t)p1, w2 = (uint64_t)(p1 >> 64);
  if (vn == cn) {                                                         // q - w as q + ~w + 1
    w0 = ~w0;
    w1 = ~w1;
    w2 = ~w2;
  }
  const unsigned __int128 a0 = (unsigned __int128)q_lo + w0 + (vn == cn ? 1u : 0u);
  const unsigned __int128 a1 = (unsigned __int128)q_hi + w1 + (uint64_t)(a0 >> 64);
  const uint64_t a2 = q_x + w2 + (uint64_t)(a1 >> 64);
  const double q = __fma_rn(__fma_rn((double)a2, kTwo64, (double)(uint64_t)a1), kTwo64, (double)(uint64_t)a0);
  const double rd = (double)r, md = math::div(rd, cnt);
  return frame_result<SH>(cnt, F, P + c, md, __fma_rn(-rd, md, q));
}
template <int SH>
__device__ __forceinline__ moments<double> frame_moments(int n, uint32_t F, int64_t P, int64_t s_hi, uint64_t s_lo, uint32_t q_x,
                                                         uint64_t q_hi, uint64_t q_lo)
{
  const double cnt = (double)n;
  const bool neg = s_hi < 0;
  const uint64_t lo = neg ? 0ull - s_lo : s_lo;
  const uint64_t hi = neg ? ~(uint64_t)s_hi + (s_lo == 0ull ? 1ull : 0ull) : (uint64_t)s_hi;
  const double mag = __fma_rn((double)hi, kTwo64, (double)lo), q = __fma_rn(__fma_rn((double)q_x, kTwo64, (double)q_hi), kTwo64, (double)q_lo);
  const double md = math::div(mag, cnt), m2 = __fma_rn(-mag, md, q);
  // m2 below a quarter of q, or negative (the bits compare as integers)
  if ((int64_t)f64i::bits(m2) + (2ll << 52) < (int64_t)f64i::bits(q)) return frame_recentred<SH>(n, F, P, s_hi, s_lo, q_x, q_hi, q_lo);
  return frame_result<SH>(cnt, F, P, neg ? -md : md, m2);
}

// var / stdev of doubles: the lane keeps its values' sum and their squared
// distances from a pivot P (the first block's mean) as exact integers in one
// fixed point frame, two bits above the first block's largest exponent.  A
// value costs some 28 integer instructions and no double ones (three on the
// double pipe, 48 clocks a warp, in the blockwise two-pass form); a value
// beyond the frame, or 512 values, closes it: its count, mean and M2 become
// doubles (frame_moments) and merge into the state.  (The frame's unit is at most
// an eighth of its largest value's ulp, and cuts bits of values below an eighth of
// that one only, beside which M2 is at least a third of its square: the cut moves
// M2 by less than 2^-50 of itself.)
template <bool W1, bool SD, class E> struct block_acc<op_moments<W1, SD>, double, E> {
  static constexpr bool value = true;
  using Op = op_moments<W1, SD>;
  using S = moments<double>;
  static constexpr int SH = 5;
  int n = 0;                       // values in the frame
  uint32_t F;                      // its exponent
  int64_t P;                       // pivot, in the frame's units
  int64_t s_hi;                    // sum of the values less P (128 bits)
  uint64_t s_lo, q_hi, q_lo;       // sum of their squares (128 bits)

  template <int N> __device__ __forceinline__ void add(S& a, const double (&x)[N])
  {
    static_assert(N <= 16 && (N & (N - 1)) == 0, "block of at most 16 values");
    const uint32_t f = f64i::max_exponent(x);
    if (n && (f > F || n > 512 - N)) flush(a);
    if (f >= 2000u) {                                      // no unit for them: value by value
#pragma unroll
      for (int i = 0; i < N; ++i) Op::add(a, x[i]);
      return;
    }
    int64_t v[N], bs = 0;
    const bool first = n == 0;
    if (first) F = (f > 64u ? f : 64u) + 2u;               // squares of smaller values underflow to 0 anyway
#pragma unroll
    for (int i = 0; i < N; ++i) {                          // below 2^58 in magnitude
      v[i] = f64i::to_fixed<SH>(x[i], F);
      bs += v[i];
    }
    if (first) {
      P = bs / N;
      s_hi = 0;
      s_lo = q_hi = q_lo = 0ull;
    }
    bs -= P * N;
    uint64_t c2 = 0ull, c1 = 0ull, c0 = 0ull;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      int64_t d = v[i] - P;                                // below 2^59
      d = d < 0 ? -d : d;
      const uint32_t lo = (uint32_t)d & 0x3fffffffu, hi = (uint32_t)(d >> 30);
      c2 += f64i::wide(hi, hi);                            // sums of 16: below 2^62, 2^63 and 2^64
      c1 += f64i::wide(hi, lo);
      c0 += f64i::wide(lo, lo);
    }
    // (s_hi:s_lo) += bs; (q_hi:q_lo) += c2 2^60 + c1 2^31 + c0
    const uint64_t t = s_lo + (uint64_t)bs;
    s_hi += (bs >> 63) + (t < s_lo ? 1 : 0);
    s_lo = t;
    add_q(c2 >> 4, c2 << 60);
    add_q(c1 >> 33, c1 << 31);
    add_q(0ull, c0);
    n += N;
  }
  __device__ __forceinline__ void add_q(uint64_t hi, uint64_t lo)
  {
    const uint64_t t = q_lo + lo;
    q_hi += hi + (t < lo ? 1ull : 0ull);
    q_lo = t;
  }
  __device__ __forceinline__ void flush(S& a)
  {
    if (n) a = closed(a, n, F, P, s_hi, s_lo, q_hi, q_lo);
    n = 0;
  }
  static __device__ __noinline__ S closed(S a, int n, uint32_t F, int64_t P, int64_t s_hi, uint64_t s_lo, uint64_t q_hi,
                                          uint64_t q_lo)
  {
    return Op::merge(a, frame_moments<SH>(n, F, P, s_hi, s_lo, 0u, q_hi, q_lo));
  }
};

// The same for a whole warp folding one segment (k_inner): the frame, its pivot
// and its closing are the warp's, the lanes' sums meet as integers, and a trip
// may be ragged (values a lane does not have add nothing), so no value and no
// lane costs a double operation of its own.
template <class Op, int N> struct warp_frame {
  using S = moments<double>;
  static constexpr int SH = 5, LOG = N == 16 ? 4 : (N == 8 ? 3 : (N == 4 ? 2 : -1));
  static_assert(LOG > 0, "4, 8 or 16 values a lane");
  int n = 0;                       // values of this lane in the frame
  bool open = false;               // the warp has one
  uint32_t F;
  int64_t P, s_hi;
  uint64_t s_lo, q_hi, q_lo;
  S lone = S{0.0, 0.0, 0.0};       // values no frame takes (infinities, NaNs, the largest): this lane's
  bool any_lone = false;

  // cnt <= N values of this lane, a prefix of x whose rest is 0; called by the whole warp
  __device__ __forceinline__ void add(S& a, const double (&x)[N], int cnt)
  {
    while (!(open && trip(x, cnt))) {
      // no frame, or not this one: a value above it, or too many values in it
      if (open) close(a);
      uint32_t f = 0u;
#pragma unroll
      for (int i = 0; i < N; ++i) {
        const uint32_t h = f64i::abs_hi(x[i]);
        f = h > f ? h : f;
      }
      f = __reduce_max_sync(0xffffffffu, f >> 20);
      if (f >= 2000u) {
#pragma unroll 1
        for (int i = 0; i < cnt; ++i) Op::add(lone, x[i]);
        any_lone = true;
        return;
      }
      F = (f > 64u ? f : 64u) + 2u;                        // squares of smaller values underflow to 0 anyway
      int64_t bs = 0;
#pragma unroll
      for (int i = 0; i < N; ++i) bs += f64i::to_fixed<SH>(x[i], F);
      const int total = (int)__reduce_add_sync(0xffffffffu, (unsigned)cnt);
      P = bs >> (5 + LOG);                                 // the pivot: the trip's mean (roughly, if it is ragged)
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) P += __shfl_xor_sync(0xffffffffu, P, off);
      if (total < 32 * N) P = (int64_t)((float)P * ((float)(32 * N) / (float)total));
      s_hi = 0;
      s_lo = q_hi = q_lo = 0ull;
      n = 0;
      open = true;
    }
  }
  // The trip's values into the open frame; false (and nothing added) if the warp
  // has one above it or a lane has no room.  The ALU pipe bounds it (two cycles an
  // instruction of a warp), hence: no running maximum, the shifts' signs tell
  // (they are below 2^31); the sign by x ^ s - s in the subtraction of the pivot;
  // differences left signed, as high * low then only needs a signed product; no
  // selection of the values a lane has: what zeros in their place added is taken
  // out.  10001 x 777 (single elements): 40.6 us before, with twice the
  // segments 35.3; 512 x 4096: 17.1 and 13.9; 4096 x 4096: 50.5 and 52.8 (8 values
  // a trip in 80 registers: 34.3, 14.0 and 59.3).
  __device__ __forceinline__ bool trip(const double (&x)[N], int cnt)
  {
    int64_t bs = 0, c2 = 0, c1 = 0;
    uint64_t c0 = 0ull;
    uint32_t above = 0u;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const uint64_t u = f64i::bits(x[i]);
      const uint32_t h = (uint32_t)(u >> 32), sh = F - ((h << 1) >> 21);
      const int64_t sg = (int32_t)h >> 31;
      const uint64_t m = ((uint64_t)((h & 0xfffffu) | 0x100000u) << 32 | (uint32_t)u) << SH;
      above |= sh;
      const int64_t d = ((int64_t)f64i::shr64(m, sh) ^ sg) - sg - P;           // below 2^59
      const int32_t lo = (int32_t)((uint32_t)d & 0x3fffffffu), hi = (int32_t)(d >> 30);
      bs += d;
      c2 += (int64_t)hi * hi;                              // sums of 16: below 2^62, 2^63 and 2^64
      c1 += (int64_t)hi * lo;
      c0 += (uint64_t)((int64_t)lo * lo);
    }
    if (__any_sync(0xffffffffu, (int32_t)above < 0 || n > 512 - N)) return false;
    if (cnt < N) {
      const int64_t k = N - cnt, d = -P;
      const int32_t lo = (int32_t)((uint32_t)d & 0x3fffffffu), hi = (int32_t)(d >> 30);
      bs -= k * d;
      c2 -= k * ((int64_t)hi * hi);
      c1 -= k * ((int64_t)hi * lo);
      c0 -= (uint64_t)k * (uint64_t)((int64_t)lo * lo);
    }
    const uint64_t t = s_lo + (uint64_t)bs;
    s_hi += (bs >> 63) + (t < s_lo ? 1 : 0);
    s_lo = t;
    add_q((uint64_t)(c2 >> 4), (uint64_t)c2 << 60);
    add_q((uint64_t)(c1 >> 33), (uint64_t)c1 << 31);
    add_q(0ull, c0);
    n += cnt;
    return true;
  }
  __device__ __forceinline__ void add_q(uint64_t hi, uint64_t lo)
  {
    const uint64_t t = q_lo + lo;
    q_hi += hi + (t < lo ? 1ull : 0ull);
    q_lo = t;
  }
  // Sum the lanes' integers (the squares in 160 bits) and merge; every lane gets the result.
  __device__ __forceinline__ void close(S& a)
  {
    a = closed(a, n, F, P, s_hi, s_lo, q_hi, q_lo);
    open = false;
    n = 0;
  }
  static __device__ __noinline__ S closed(S a, int n, uint32_t F, int64_t P, int64_t s_hi, uint64_t s_lo, uint64_t q_hi,
                                          uint64_t q_lo)
  {
    uint32_t q_x = 0u;
#pragma unroll 1
    for (int off = 16; off > 0; off >>= 1) {
      const uint64_t sl = __shfl_xor_sync(0xffffffffu, s_lo, off), ql = __shfl_xor_sync(0xffffffffu, q_lo, off);
      const int64_t sh = __shfl_xor_sync(0xffffffffu, s_hi, off);
      const uint64_t qh = __shfl_xor_sync(0xffffffffu, q_hi, off);
      const uint32_t qx = __shfl_xor_sync(0xffffffffu, q_x, off);
      n += __shfl_xor_sync(0xffffffffu, n, off);
      s_lo += sl;
      s_hi += sh + (s_lo < sl ? 1 : 0);
      q_lo += ql;
      const uint64_t c = q_lo < ql ? 1ull : 0ull, h1 = q_hi + qh, h2 = h1 + c;
      q_x += qx + (h1 < qh ? 1u : 0u) + (h2 < c ? 1u : 0u);
      q_hi = h2;
    }
    return Op::merge(a, frame_moments<SH>(n, F, P, s_hi, s_lo, q_x, q_hi, q_lo));
  }
};
template <class Op, class T> struct warp_framed { static constexpr bool value = false; };
template <bool W1, bool SD> struct warp_framed<op_moments<W1, SD>, double> { static constexpr bool value = true; };

// Resident blocks asked for: four (64 registers; six for short columns, which
// take few loads and wait for them), two where a lane keeps the
// integer frame of var/stdev beside its 16 values.
template <class Op, class T, int U> struct fold_min_blocks { static constexpr int value = U <= 4 ? 6 : 4; };
template <int FIN, int U> struct fold_min_blocks<op_sum<false, FIN>, double, U> { static constexpr int value = 4; };   // 512 x 4096: 5.5 us, 7.6 with six
template <bool W1, bool SD, int U> struct fold_min_blocks<op_moments<W1, SD>, double, U> { static constexpr int value = U <= 4 ? 3 : 2; };

template <class Op, class T> using out_of = typename Op::template out_t<T>;

// Butterfly over the warp; every lane ends with the same value.
template <class Op, class T> __device__ __forceinline__ state_of<Op, T> warp_merge(state_of<Op, T> a)
{
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    state_of<Op, T> o = Op::shfl(a, off);
    // combine in lane order so every lane computes the same value
    a = ((threadIdx.x & 31) & off) ? Op::merge(o, a) : Op::merge(a, o);
  }
  return a;
}

// Merge n partials p[0], p[stride], ... in index order, with 8 loads in
// flight at a time (the merge is at the tail of the kernel, where serial L2
// round trips would show).
template <class Op, class T, int N = 8>
__device__ __forceinline__ state_of<Op, T> merge_partials(const state_of<Op, T>* p, size_t n, size_t stride)
{
  state_of<Op, T> m = Op::template init<T>();
  size_t q = 0;
#pragma unroll 1
  for (; q + N <= n; q += N) {
    state_of<Op, T> v[N];
#pragma unroll
    for (int k = 0; k < N; ++k) v[k] = Op::ldcg(p + (q + k) * stride);
#pragma unroll
    for (int k = 0; k < N; ++k) m = Op::merge(m, v[k]);
  }
#pragma unroll 1
  for (; q < n; ++q) m = Op::merge(m, Op::ldcg(p + q * stride));
  return m;
}

// Folds of zero elements: every output is finish(neutral).
template <class Op, class T>
__global__ void __launch_bounds__(256) k_fold_empty(out_of<Op, T>* __restrict__ out, size_t count)
{
  nt2cuda::mem::pdl_begin();
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += (size_t)gridDim.x * blockDim.x)
    out[i] = Op::finish(Op::template init<T>(), 0);
}

// ------------------------------------------------------------ inner fold
// Work unit: one warp reduces the segment [r0, r1) of column j, where the
// column is split into `splits` segments of `seg` elements (seg a multiple
// of 32*V).  With splits > 1 the warp writes its partial to scratch and the
// last warp of the column combines the column's partials in segment order.
struct inner_shape {
  size_t rows, cols, seg, splits;
};

// fold_min_blocks: left to itself the compiler keeps 48 registers, 32 where a
// lane loads single elements; 64 leave room for more of a trip's loads at once
// (though not for all of 16 times 16 bytes): sum(A,1) of 8192 x 4096 floats
// 24.5 us, now 21.5; 300001 x 50, single elements, 27.8 us, now 14.8.
template <class Op, int V, int U, class T, class E>
__global__ void __launch_bounds__(256, (fold_min_blocks<Op, T, U>::value)) k_inner(E e, inner_shape sh, out_of<Op, T>* __restrict__ out,
                                               state_of<Op, T>* __restrict__ partials, unsigned* __restrict__ counters)
{
  const int lane = threadIdx.x & 31;
  const size_t warps_total = (size_t)gridDim.x * (blockDim.x >> 5);
  const size_t units = sh.cols * sh.splits;
  {
    // while the previous grid drains, have the L2 fetch the lines of this
    // warp's first U loads (one prefetch per 128-byte line)
    const size_t w = (size_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    constexpr int LANES_PER_LINE = (V * (int)sizeof(T)) >= 128 ? 1 : 128 / (V * (int)sizeof(T));
    if (w < units && V > 1 && lane % LANES_PER_LINE == 0) {
      const size_t j = sh.splits == 1 ? w : w / sh.splits, r0 = (w - j * sh.splits) * sh.seg;
      const size_t r1 = (r0 + sh.seg < sh.rows) ? r0 + sh.seg : sh.rows;
      const size_t g1 = r1 / V;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const size_t g = r0 / V + lane + (size_t)u * 32;
        if (g < g1) prefetch_terms(e, j * sh.rows + g * V);
      }
    }
  }
  nt2cuda::mem::pdl_begin();
  for (size_t w = (size_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); w < units; w += warps_total) {
    const size_t j = sh.splits == 1 ? w : w / sh.splits, sp = w - j * sh.splits;   // a 64-bit division is long
    const size_t r0 = sp * sh.seg;
    const size_t r1 = (r0 + sh.seg < sh.rows) ? r0 + sh.seg : sh.rows;
    const size_t base = j * sh.rows;
    constexpr bool BLK = block_acc<Op, T, E>::value;
    block_acc<Op, T, E> ba;
    state_of<Op, T> a[V];
#pragma unroll
    for (int l = 0; l < V; ++l) a[l] = Op::template init<T>();
    const size_t g0 = r0 / V, g1 = r1 / V;   // r0 is a multiple of V
    if constexpr (warp_framed<Op, T>::value) {
      constexpr int N = U * V;
      warp_frame<Op, N> wf;
      state_of<Op, T> t = Op::template init<T>();
      // the V-groups, and (r1 % V != 0 only at a column's end) the ragged rest, one value per lane
      for (size_t g = g0; g < g1; g += (size_t)U * 32) {
        T x[N] = {};
        int have = N;
        if (g + (size_t)U * 32 <= g1) {
          regs<E, V> rr[U];
#pragma unroll
          for (int u = 0; u < U; ++u) rr[u].template load<true>(e, base + (g + (size_t)u * 32 + lane) * V);
#pragma unroll
          for (int u = 0; u < U; ++u)
#pragma unroll
            for (int l = 0; l < V; ++l) x[u * V + l] = (T)rr[u].template get<false>(e, l);
        } else {
          have = 0;
#pragma unroll
          for (int u = 0; u < U; ++u)
            if (g + (size_t)u * 32 + lane < g1) {
              regs<E, V> rr;
              rr.template load<true>(e, base + (g + (size_t)u * 32 + lane) * V);
#pragma unroll
              for (int l = 0; l < V; ++l) x[u * V + l] = (T)rr.template get<false>(e, l);
              have += V;
            }
        }
        wf.add(t, x, have);
      }
      for (size_t r = g1 * V; r < r1; r += 32) {
        T x[N] = {};
        const int have = r + lane < r1 ? 1 : 0;
        if (have) {
          regs<E, 1> rr;
          rr.template load<false>(e, base + r + lane);
          x[0] = (T)rr.template get<false>(e, 0);
        }
        wf.add(t, x, have);
      }
      if (wf.open) wf.close(t);
      if (wf.any_lone) t = Op::merge(t, warp_merge<Op, T>(wf.lone));
      a[0] = t;
    }
    // full V-groups
    size_t g = warp_framed<Op, T>::value ? g1 : g0 + lane;
    if constexpr (!warp_framed<Op, T>::value) {
    for (; g + (size_t)(U - 1) * 32 < g1; g += (size_t)U * 32) {
      regs<E, V> rr[U];
#pragma unroll
      for (int u = 0; u < U; ++u) rr[u].template load<true>(e, base + (g + (size_t)u * 32) * V);
      if constexpr (BLK) {
        T blk[U * V];
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
          for (int l = 0; l < V; ++l) blk[u * V + l] = (T)rr[u].template get<false>(e, l);
        ba.add(a[0], blk);
      } else {
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
          for (int l = 0; l < V; ++l) Op::add(a[l], (T)rr[u].template get<false>(e, l));
      }
    }
    // what is left of the segment: four groups at a time, then at most three
    if constexpr (U > 4) {
#pragma unroll 1
      for (; g + (size_t)3 * 32 < g1; g += (size_t)4 * 32) {
        regs<E, V> rr[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) rr[u].template load<true>(e, base + (g + (size_t)u * 32) * V);
        if constexpr (BLK) {
          T blk[4 * V];
#pragma unroll
          for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int l = 0; l < V; ++l) blk[u * V + l] = (T)rr[u].template get<false>(e, l);
          ba.add(a[0], blk);
        } else {
#pragma unroll
          for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int l = 0; l < V; ++l) Op::add(a[l], (T)rr[u].template get<false>(e, l));
        }
      }
    }
    {
      regs<E, V> rr[3];
#pragma unroll
      for (int u = 0; u < 3; ++u)
        if (g + (size_t)u * 32 < g1) rr[u].template load<true>(e, base + (g + (size_t)u * 32) * V);
      // a loop over the trips the warp has, the loaded values moving up: unrolled,
      // each add becomes a predicated one, and those that are off still take
      // their turn on the double pipe
      const size_t gw = g - lane;
#pragma unroll 1
      for (size_t q = gw; q < g1; q += 32) {
        if (q + lane < g1) {
#pragma unroll
          for (int l = 0; l < V; ++l) Op::add(a[l], (T)rr[0].template get<false>(e, l));
        }
        rr[0] = rr[1];
        rr[1] = rr[2];
      }
    }
    if constexpr (BLK) ba.flush(a[0]);
    }
    // ragged end of the segment (only when rows % V != 0 or V == 1)
    if constexpr (!warp_framed<Op, T>::value)
      for (size_t r = g1 * V + lane; r < r1; r += 32) {
        regs<E, 1> rr;
        rr.template load<false>(e, base + r);
        Op::add(a[0], (T)rr.template get<false>(e, 0));
      }
    state_of<Op, T> t = a[0];
    if constexpr (!warp_framed<Op, T>::value) {
#pragma unroll
      for (int l = 1; l < V; ++l) t = Op::merge(t, a[l]);
      t = warp_merge<Op, T>(t);
    }
    if (sh.splits == 1) {
      if (lane == 0) out[j] = Op::finish(t, sh.rows);
      continue;
    }
    unsigned last = 0;
    if (lane == 0) {
      partials[w] = t;
      __threadfence();
      unsigned prev = atomicAdd(&counters[j], 1u);
      last = (prev == (unsigned)sh.splits - 1u);
      if (last) counters[j] = 0u;   // ready for the next call on this scratch
    }
    last = __shfl_sync(0xffffffffu, last, 0);
    if (!last) continue;
    __threadfence();
    // combine the column's partials in a fixed order: lane k folds segments
    // k, k+32, ..., then the butterfly merges lanes in order
    const size_t mine = sh.splits > (size_t)lane ? (sh.splits - lane + 31) / 32 : 0;
    state_of<Op, T> c = merge_partials<Op, T>(partials + j * sh.splits + lane, mine, 32);
    c = warp_merge<Op, T>(c);
    if (lane == 0) out[j] = Op::finish(c, sh.rows);
  }
}

// Short columns (rows < 32): one thread folds one whole column.
template <class Op, class T, class E>
__global__ void __launch_bounds__(256) k_inner_short(E e, size_t rows, size_t cols, out_of<Op, T>* __restrict__ out)
{
  nt2cuda::mem::pdl_begin();
  for (size_t j = (size_t)blockIdx.x * blockDim.x + threadIdx.x; j < cols; j += (size_t)gridDim.x * blockDim.x) {
    state_of<Op, T> a = Op::template init<T>();
    for (size_t r = 0; r < rows; ++r) {
      regs<E, 1> rr;
      rr.template load<false>(e, j * rows + r);
      Op::add(a, (T)rr.template get<false>(e, 0));
    }
    out[j] = Op::finish(a, rows);
  }
}

// ------------------------------------------------------------ outer fold
// Row sums of a rows x cols column-major table.  A block owns a strip of
// 32*V rows (one V-group per lane) and a chunk of `cchunk` columns; its 8
// warps take the chunk's columns round-robin, and the block merges the
// warps' partials in warp order.  With splits > 1 the block's per-row
// partials go to scratch and the last block of the strip merges them in
// chunk order.
struct outer_shape {
  size_t rows, cols, cchunk, splits, strips;
};

// fold_min_blocks: as in k_inner (8192 x 4096 floats 24.2 us with the compiler's
// own 48 registers, now 22.5; 10001 x 777 floats 20.3, now 9.7).
template <class Op, int V, int U, class T, class E>
__global__ void __launch_bounds__(256, (fold_min_blocks<Op, T, U>::value)) k_outer(E e, outer_shape sh, out_of<Op, T>* __restrict__ out,
                                               state_of<Op, T>* __restrict__ partials, unsigned* __restrict__ counters)
{
  using S = state_of<Op, T>;
  constexpr int STRIP = 32 * V;
  __shared__ S red[8][STRIP];
  __shared__ unsigned is_last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const size_t units = sh.strips * sh.splits;
  {
    // while the previous grid drains, have the L2 fetch the lines of this
    // warp's first U loads of its first unit (one prefetch per 128-byte line)
    constexpr int LANES_PER_LINE = (V * (int)sizeof(T)) >= 128 ? 1 : 128 / (V * (int)sizeof(T));
    const size_t b = blockIdx.x;
    if (b < units && V > 1 && lane % LANES_PER_LINE == 0) {
      const size_t strip = b / sh.splits, m0 = (b % sh.splits) * sh.cchunk;
      const size_t row0 = strip * STRIP + (size_t)lane * V;
      const size_t m1 = (m0 + sh.cchunk < sh.cols) ? m0 + sh.cchunk : sh.cols;
      if (row0 + V <= sh.rows) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const size_t m = m0 + warp + (size_t)u * 8;
          if (m < m1) prefetch_terms(e, m * sh.rows + row0);
        }
      }
    }
  }
  nt2cuda::mem::pdl_begin();
  for (size_t b = blockIdx.x; b < units; b += gridDim.x) {
    const size_t strip = b / sh.splits, sp = b % sh.splits;
    const size_t row0 = strip * STRIP + (size_t)lane * V;   // first row of this lane
    const size_t m0 = sp * sh.cchunk;
    const size_t m1 = (m0 + sh.cchunk < sh.cols) ? m0 + sh.cchunk : sh.cols;
    const bool full = row0 + V <= sh.rows;
    constexpr bool BLK = block_acc<Op, T, E>::value;
    block_acc<Op, T, E> ba[V];
    S a[V];
#pragma unroll
    for (int l = 0; l < V; ++l) a[l] = Op::template init<T>();
    if (full) {
      size_t m = m0 + warp;
      for (; m + (size_t)(U - 1) * 8 < m1; m += (size_t)U * 8) {
        regs<E, V> rr[U];
#pragma unroll
        for (int u = 0; u < U; ++u) rr[u].template load<true>(e, (m + (size_t)u * 8) * sh.rows + row0);
        if constexpr (BLK) {
          // lane slot l is one row: its U values of this trip form a block
#pragma unroll
          for (int l = 0; l < V; ++l) {
            T blk[U];
#pragma unroll
            for (int u = 0; u < U; ++u) blk[u] = (T)rr[u].template get<false>(e, l);
            ba[l].add(a[l], blk);
          }
        } else {
#pragma unroll
          for (int u = 0; u < U; ++u)
#pragma unroll
            for (int l = 0; l < V; ++l) Op::add(a[l], (T)rr[u].template get<false>(e, l));
        }
      }
      if constexpr (U > 4) {
#pragma unroll 1
        for (; m + (size_t)3 * 8 < m1; m += (size_t)4 * 8) {
          regs<E, V> rr[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) rr[u].template load<true>(e, (m + (size_t)u * 8) * sh.rows + row0);
          if constexpr (BLK) {
#pragma unroll
            for (int l = 0; l < V; ++l) {
              T blk[4];
#pragma unroll
              for (int u = 0; u < 4; ++u) blk[u] = (T)rr[u].template get<false>(e, l);
              ba[l].add(a[l], blk);
            }
          } else {
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
              for (int l = 0; l < V; ++l) Op::add(a[l], (T)rr[u].template get<false>(e, l));
          }
        }
      }
      {
        regs<E, V> rr[3];
#pragma unroll
        for (int u = 0; u < 3; ++u)
          if (m + (size_t)u * 8 < m1) rr[u].template load<true>(e, (m + (size_t)u * 8) * sh.rows + row0);
#pragma unroll 1
        for (size_t q = m; q < m1; q += 8) {      // a loop, not predicated adds: see k_inner
#pragma unroll
          for (int l = 0; l < V; ++l) Op::add(a[l], (T)rr[0].template get<false>(e, l));
          rr[0] = rr[1];
          rr[1] = rr[2];
        }
      }
      if constexpr (BLK)
#pragma unroll
        for (int l = 0; l < V; ++l) ba[l].flush(a[l]);
    } else if (row0 < sh.rows) {
      for (size_t m = m0 + warp; m < m1; m += 8)
#pragma unroll
        for (int l = 0; l < V; ++l)
          if (row0 + l < sh.rows) {
            regs<E, 1> rr;
            rr.template load<false>(e, m * sh.rows + row0 + l);
            Op::add(a[l], (T)rr.template get<false>(e, 0));
          }
    }
#pragma unroll
    for (int l = 0; l < V; ++l) red[warp][lane * V + l] = a[l];
    __syncthreads();
    // thread t < STRIP merges row t of the strip over the 8 warps in order
    S rsum = Op::template init<T>();
    const size_t row = strip * STRIP + threadIdx.x;
    if (threadIdx.x < STRIP) {
      rsum = red[0][threadIdx.x];
#pragma unroll
      for (int w = 1; w < 8; ++w) rsum = Op::merge(rsum, red[w][threadIdx.x]);
    }
    if (sh.splits == 1) {
      if (threadIdx.x < STRIP && row < sh.rows) out[row] = Op::finish(rsum, sh.cols);
      __syncthreads();
      continue;
    }
    if (threadIdx.x < STRIP) partials[b * STRIP + threadIdx.x] = rsum;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
      unsigned prev = atomicAdd(&counters[strip], 1u);
      is_last = (prev == (unsigned)sh.splits - 1u);
      if (is_last) counters[strip] = 0u;
    }
    __syncthreads();
    if (is_last) {
      __threadfence();
      // merge the strip's chunks in a fixed order: the threads are 256/STRIP groups
      // over the rows, group g takes chunks g, g + G, ..., then the groups in order
      constexpr int G = 256 / STRIP;
      const int r = threadIdx.x % STRIP, g = threadIdx.x / STRIP;
      const size_t mine = sh.splits > (size_t)g ? (sh.splits - g + G - 1) / G : 0;
      red[g][r] = merge_partials<Op, T, 4>(partials + (strip * sh.splits + g) * STRIP + r, mine, (size_t)G * STRIP);
      __syncthreads();
      if (threadIdx.x < STRIP && row < sh.rows) {
        S c = red[0][threadIdx.x];
#pragma unroll
        for (int w = 1; w < G; ++w) c = Op::merge(c, red[w][threadIdx.x]);
        out[row] = Op::finish(c, sh.cols);
      }
    }
    __syncthreads();
  }
}

}  // namespace fold
}  // namespace nt2cuda
