// nt2cuda/fold_launch.cuh -- host launchers of the inner_fold and outer_fold
// kernels for any elementwise expression E (globalsum(X*Y) is
// inner_fold(node<multiplies_, term, term>, n, 1)).
// The NT2 overloads they replace are
// modules/arch/shared_memory/include/nt2/core/functions/shared_memory/inner_fold.hpp:24-63 and
// .../shared_memory/outer_fold.hpp:22-51.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include "expr.cuh"
#include "fold.cuh"
#include "launch.cuh"
#include "scratch.cuh"
#include "fold_tma.cuh"
#include <stdlib.h>
#include <string.h>
#include <algorithm>
#include <atomic>

namespace nt2cuda {
namespace fold {

inline size_t round_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

template <class E> bool expr_aligned(const E& e)
{
  bool ok = true;
  visit_expr(e, [&](ptr_span s) { if (((uintptr_t)s.p) & 15u) ok = false; }, 0);
  return ok;
}

// How inner_fold cuts columns into segments, one to a warp: into about
// `kInnerUnits` segments in all, 24 a SM with 16-byte loads and 16 with single
// elements, so that a few long columns fill the chip too (3333333 x 1 floats:
// 44 us with segments of 16384, 10.5 with 16 a SM), but never below eight
// loads a lane, and at most kInnerSplits to a column, as one warp merges them.
// The cut depends on the table's shape alone (and on whether the call is captured,
// see captured_cut): results are reproducible.
// (var/stdev of doubles: 16 a SM in either case, what their 128 registers leave
// room for; 70000 x 111: 46.9 us with 8, 40.7 with 16, 41.6 with 24.)
constexpr size_t kInnerUnits = 24 * kSms, kInnerUnitsScalar = 16 * kSms, kInnerSplits = 16 * kSms;
template <class Op, class T> inline size_t inner_seg(size_t rows, size_t cols, bool vec)
{
  const size_t lanes = vec ? 32 * (16 / sizeof(T)) : 32;
  const size_t units = vec && !warp_framed<Op, T>::value ? kInnerUnits : kInnerUnitsScalar;
  size_t splits = (units + cols / 2) / cols;              // rounded: half a segment more or less a column
  if (splits < 1) splits = 1;
  if (splits > kInnerSplits) splits = kInnerSplits;
  size_t seg = round_up((rows + splits - 1) / splits, lanes);
  return seg < lanes * 8 ? lanes * 8 : seg;
}

// Which kernels serve the folds of a table or of a product of two tables:
//   0 (auto): TMA-staged for long columns (inner_fold, rows >= 2^16), the
//             register-pipelined kernels otherwise;
//   1 (simt): always the register-pipelined kernels;
//   2 (tma):  TMA-staged wherever the tables allow it (16-byte aligned, whole
//             vectors long; outer_fold from 256 rows).
// The initial value comes from NT2CUDA_FOLD_PATH ("auto", "simt", "tma").
inline std::atomic<int>& fold_path()
{
  static std::atomic<int> p([] {
    const char* e = getenv("NT2CUDA_FOLD_PATH");
    if (e && !strcmp(e, "simt")) return 1;
    if (e && !strcmp(e, "tma")) return 2;
    return 0;
  }());
  return p;
}

template <class T> struct tma_terms { static constexpr int n = 0; };
template <class T> struct tma_terms<term<T>> { static constexpr int n = 1; };
template <class T> struct tma_terms<node<tag::multiplies_, term<T>, term<T>>> { static constexpr int n = 2; };

template <class T> inline const T* first_term(const term<T>& t) { return t.p; }
template <class T> inline const T* first_term(const node<tag::multiplies_, term<T>, term<T>>& n) { return n.a.p; }
template <class T> inline const T* second_term(const term<T>&) { return nullptr; }
template <class T> inline const T* second_term(const node<tag::multiplies_, term<T>, term<T>>& n) { return n.b.p; }

// Loads of a lane's trip in the register-pipelined kernels: 16, or 8 where a
// trip's values form a block (block_acc): its values stay in registers.
template <class Op, class T, class E> struct fold_unroll {
  static constexpr int value = block_acc<Op, T, E>::value ? 8 : 16;
};
// outer_fold keeps V rows' states per lane: var/stdev of floats there take 4 columns a trip
template <class Op, class T, class E> struct outer_unroll { static constexpr int value = fold_unroll<Op, T, E>::value; };
template <bool W1, bool SD, class E> struct outer_unroll<op_moments<W1, SD>, float, E> { static constexpr int value = 4; };
// Tables whose rows or alignment rule out 16-byte loads: one element per lane
// and load, so 16 loads a trip again.
constexpr int kScalarUnroll = 16;
constexpr size_t kOuterUnits = 4 * kSms;

// Segments of inner_fold under capture (captured_cut): 128 loads of 16 bytes a lane,
// or 16 bulk-copy tiles where a column of double var/stdev would otherwise be staged.
template <class Op, class T, class E> inline size_t inner_wide(size_t rows, bool vec)
{
  constexpr size_t VV = 16 / sizeof(T), seg = 32 * VV * 128;
  if (warp_framed<Op, T>::value && tma_terms<E>::n > 0 && vec && rows >= ((size_t)1 << 16))
    return (size_t)inner_tile<T>() * 16;
  return seg;
}

template <class Op, class T> cudaError_t fold_empty(out_of<Op, T>* out, size_t count, cudaStream_t s)
{
  void* args[] = {&out, &count};
  return launch_persistent(k_fold_empty<Op, T>, count, 256, 1, s, args);
}

// inner_fold with operation Op (op_sum<COMP>, op_val, op_logic, op_moments).
template <class Op, class T, class E>
cudaError_t inner_fold(const E& e, size_t rows, size_t cols, out_of<Op, T>* out, cudaStream_t s)
{
  using S = state_of<Op, T>;
  if constexpr (tma_terms<E>::n > 0) {
    constexpr size_t VV = 16 / sizeof(T);
    // auto: long columns only; a short column's tiles are too few to amortise the block barriers
    const int path = fold_path().load(std::memory_order_relaxed);
    const size_t min_rows = path == 2 ? 32 : ((size_t)1 << 16);
    // (var/stdev of doubles: the register-pipelined kernel, whose integer frames
    // leave the staged one a single block per SM)
    constexpr bool staged = !(std::is_same<S, moments<double>>::value);
    if (path != 1 && (staged || path == 2) && rows >= min_rows && cols > 0 && out && rows % VV == 0 && expr_aligned(e) &&
        std::is_same<typename value_of<E>::type, T>::value)
      return inner_fold_tma<Op, T>(first_term(e), second_term(e), rows, cols, out, s);
  }
  if (cols == 0) return cudaSuccess;
  if (!out) return cudaErrorInvalidValue;
  if (rows == 0) return fold_empty<Op, T>(out, cols, s);
  if (rows < 32) {
    size_t ee = cols;
    E ec = e;
    out_of<Op, T>* o = out;
    void* args[] = {&ec, &rows, &ee, &o};
    return (launch_persistent(k_inner_short<Op, T, E>, cols, 256, 4, s, args));
  }
  constexpr int VV = 16 / (int)sizeof(T);
  const bool vec = expr_aligned(e) && rows % VV == 0;
  inner_shape sh;
  sh.rows = rows;
  sh.cols = cols;
  sh.seg = inner_seg<Op, T>(rows, cols, vec);
  sh.splits = (rows + sh.seg - 1) / sh.seg;
  const size_t wide_seg = inner_wide<Op, T, E>(rows, vec), wide = (rows + wide_seg - 1) / wide_seg;
  if (captured_cut(sh.splits, wide, s) != sh.splits) {
    sh.seg = wide_seg;
    sh.splits = wide;
  }
  void* partials = nullptr;
  unsigned* counters = nullptr;
  const cudaError_t st = fold_scratch(s, cols, sh.splits, wide, sizeof(S), &counters, &partials);
  if (st != cudaSuccess) return st;
  const size_t units = cols * sh.splits;
  E ec = e;
  out_of<Op, T>* o = out;
  void* args[] = {&ec, &sh, &o, &partials, &counters};
  // launch_persistent counts threads; a unit is one warp.  Columns of at most
  // eight loads a lane take the kernel with four a trip.
  if (rows <= (size_t)32 * (vec ? VV : 1) * 8) {
    if (vec) return (launch_persistent(k_inner<Op, VV, 4, T, E>, units * 32, 128, 4, s, args));
    return (launch_persistent(k_inner<Op, 1, 4, T, E>, units * 32, 128, 4, s, args));
  }
  if (vec) return (launch_persistent(k_inner<Op, VV, fold_unroll<Op, T, E>::value, T, E>, units * 32, 128, 4, s, args));
  return (launch_persistent(k_inner<Op, 1, kScalarUnroll, T, E>, units * 32, 128, 4, s, args));
}

template <class Op, class T, class E>
cudaError_t outer_fold(const E& e, size_t rows, size_t cols, out_of<Op, T>* out, cudaStream_t s)
{
  using S = state_of<Op, T>;
  if constexpr (tma_terms<E>::n == 1) {
    constexpr size_t VV = 16 / sizeof(T);
    if (fold_path().load(std::memory_order_relaxed) == 2 && rows >= 256 && cols > 0 && out && rows % VV == 0 &&
        expr_aligned(e) && rows < ((size_t)1 << 31) && cols < ((size_t)1 << 31)) {
      cudaError_t r = outer_fold_tma<Op, T>(first_term(e), rows, cols, out, s);
      if (r != cudaErrorNotSupported) return r;
    }
  }
  if (rows == 0) return cudaSuccess;
  if (!out) return cudaErrorInvalidValue;
  if (cols == 0) return fold_empty<Op, T>(out, rows, s);
  constexpr int VV = 16 / (int)sizeof(T);
  const bool vec = expr_aligned(e) && rows % VV == 0;
  const int V = vec ? VV : 1;
  const size_t STRIP = (size_t)32 * V;
  outer_shape sh;
  sh.rows = rows;
  sh.cols = cols;
  sh.strips = (rows + STRIP - 1) / STRIP;
  // as many chunks as keep the blocks within four a SM: one wave, every
  // block at once (8192 x 4096 floats in 640 blocks takes 29.8 us); under capture
  // (captured_cut) whole 64 columns in about 512 blocks.  The split depends only on
  // the shape, so results stay reproducible.
  const size_t want = sh.strips < kOuterUnits ? kOuterUnits / sh.strips : 1, wide_want = (512 + sh.strips - 1) / sh.strips;
  const size_t chunk = round_up((cols + want - 1) / want, 8), wide_chunk = round_up((cols + wide_want - 1) / wide_want, 64);
  sh.cchunk = chunk < 64 ? 64 : chunk;
  sh.splits = (cols + sh.cchunk - 1) / sh.cchunk;
  const size_t wide = (cols + wide_chunk - 1) / wide_chunk;
  if (captured_cut(sh.splits, wide, s) != sh.splits) {
    sh.cchunk = wide_chunk;
    sh.splits = wide;
  }
  void* partials = nullptr;
  unsigned* counters = nullptr;
  const cudaError_t st = fold_scratch(s, sh.strips, sh.splits, wide, sizeof(S), &counters, &partials, STRIP);
  if (st != cudaSuccess) return st;
  const size_t units = sh.strips * sh.splits;
  E ec = e;
  out_of<Op, T>* o = out;
  void* args[] = {&ec, &sh, &o, &partials, &counters};
  if (vec) return (launch_persistent(k_outer<Op, VV, outer_unroll<Op, T, E>::value, T, E>, units * 256, 256, 4, s, args));
  return (launch_persistent(k_outer<Op, 1, kScalarUnroll, T, E>, units * 256, 256, 4, s, args));
}

}  // namespace fold
}  // namespace nt2cuda

