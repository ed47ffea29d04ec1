// nt2cuda/scan_launch.cuh -- host launchers of the scan kernels (scan.cuh):
// inner_scan (along dim 1) and outer_scan (along dim 2) of a column-major
// table, out-of-place or in place.  The NT2 overloads they replace are
// modules/arch/shared_memory/include/nt2/core/functions/shared_memory/{inner,outer}_scan.hpp.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include "launch.cuh"
#include "scan.cuh"
#include "scratch.cuh"
#include "wait_status.cuh"

namespace nt2cuda {
namespace scan {

inline size_t align256(size_t b) { return (b + 255) / 256 * 256; }

// Scratch of the look-back over `tiles` tiles: ticket and error word, flags,
// aggregates, inclusive prefixes.
constexpr size_t kScanHead = 256;
inline size_t flag_bytes(size_t tiles) { return align256(tiles * sizeof(unsigned)); }
template <class Op, class T> inline size_t side_bytes(size_t tiles) { return align256(tiles * carry_bytes<Op, T>()); }
template <class Op, class T> inline size_t lookback_scratch(size_t tiles)
{
  return kScanHead + flag_bytes(tiles) + 2 * side_bytes<Op, T>(tiles);
}

// The streamed scan of long float columns (k_scan_stream).  cudaErrorNotSupported,
// before anything is launched, when it does not apply.
// At least a tile for each SM (1.9 million floats 18.2 us before, 15.1),
// and at most an eighth of padding in the columns' last tiles
// (16384 x 1000, a third of whose tiles' rows would be padding: 39.7 against 50).
constexpr size_t kStreamTiles = kSms;
template <class Op, class T> struct streamed { static constexpr bool value = false; };
template <bool COMP> struct streamed<fold::op_sum<COMP>, float> { static constexpr bool value = true; static constexpr bool comp = COMP; };
// first, wait_rounds and polls are for the timeout self-test: the tile handed out
// first, and the bounds of the waits.
template <bool COMP>
cudaError_t inner_scan_stream(const float* x, float* y, size_t rows, size_t cols, cudaStream_t s, unsigned first = 0,
                              uint32_t wait_rounds = tma::kMaxRounds, uint32_t polls = kSpinMax)
{
  if (rows < kStreamTile || rows / 32 >= ((size_t)1 << 31) || cols >= ((size_t)1 << 31) || (cols > 1 && rows % 4) ||
      (((uintptr_t)x | (uintptr_t)y) & 15u))
    return cudaErrorNotSupported;
  stream_shape sh;
  sh.rows = rows;
  sh.cols = cols;
  sh.tiles_per_col = (rows / 32 + kStreamRows - 1) / kStreamRows;
  sh.tiles = sh.tiles_per_col * cols;
  sh.wait_rounds = wait_rounds;
  sh.polls = polls;
  if (sh.tiles < kStreamTiles || sh.tiles_per_col * kStreamTile > rows + rows / 8) return cudaErrorNotSupported;
  PFN_cuTensorMapEncodeTiled_v12000 encode = tma::tensor_map_encoder();
  if (!encode) return cudaErrorNotSupported;
  CUtensorMap xmap, ymap;
  const cuuint64_t gdim[3] = {32, (cuuint64_t)(rows / 32), (cuuint64_t)cols};
  const cuuint64_t gstride[2] = {128, (cuuint64_t)(cols > 1 ? rows * sizeof(float) : (rows / 32) * 128)};
  const cuuint32_t box[3] = {32, kStreamRows / 2, 1};
  const cuuint32_t estride[3] = {1, 1, 1};
  if (encode(&xmap, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, (void*)x, gdim, gstride, box, estride, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS ||
      encode(&ymap, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, (void*)y, gdim, gstride, box, estride, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return cudaErrorNotSupported;
  // scratch: ticket | aggregates, all kStreamEmpty; never less than the look-back
  // would take, so that a misaligned column of this shape can be captured after it
  using K = scan_tiles<fold::op_sum<COMP>, float>;
  void* scratch = nullptr;
  const size_t head = kScanHead, sbytes = sh.tiles * kStreamWords * sizeof(unsigned long long);
  const size_t other = lookback_scratch<fold::op_sum<COMP>, float>((rows + K::TILE - 1) / K::TILE * cols);
  cudaError_t e = nt2cuda::stream_scratch(s, head + sbytes > other ? head + sbytes : other, &scratch, 1);
  if (e != cudaSuccess) return e;
  unsigned long long* ticket = (unsigned long long*)scratch;
  unsigned long long* agg = (unsigned long long*)((char*)scratch + head);
  if ((e = cudaMemsetAsync(scratch, 0x7f, head + sbytes, s)) != cudaSuccess) return e;
  if (first && (e = cudaMemsetAsync(scratch, 0x7f + (int)first, 1, s)) != cudaSuccess) return e;
  auto k = k_scan_stream<COMP>;
  if ((e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kStreamSmem)) != cudaSuccess) return e;
  size_t grid = (size_t)sm_count();
  if (grid > sh.tiles) grid = sh.tiles;
  void* args[] = {(void*)&xmap, (void*)&ymap, (void*)&x, (void*)&y, (void*)&sh, (void*)&ticket, (void*)&agg};
  return launch_dependent(k, grid, kStreamThreads, s, args, kStreamSmem);
}

template <class Op, class T>
cudaError_t inner_scan(const T* x, T* y, size_t rows, size_t cols, cudaStream_t s)
{
  using S = state_of<Op, T>;
  if (!rows || !cols) return cudaSuccess;
  if (rows <= 64) {
    void* args[] = {(void*)&x, (void*)&y, (void*)&rows, (void*)&cols};
    return launch_persistent(k_scan_inner_short<Op, T>, cols, 256, 2, s, args);
  }
  if constexpr (streamed<Op, T>::value) {
    const cudaError_t e = inner_scan_stream<streamed<Op, T>::comp>(x, y, rows, cols, s);
    if (e != cudaErrorNotSupported) return e;
  }
  // columns of one 32 KB tile: a single pass without look-back; other longer ones:
  // 64 KB tiles chained by the look-back, aggregate then rescan from L2
  const bool one_pass = rows <= (size_t)tile<T>();
  const size_t TILE = one_pass ? (size_t)tile<T>() : scan_tiles<Op, T>::TILE;
  inner_shape sh;
  sh.rows = rows;
  sh.cols = cols;
  sh.tiles_per_col = (rows + TILE - 1) / TILE;
  sh.tiles = sh.tiles_per_col * cols;
  // scratch: ticket, error word, flags | aggregates | inclusive prefixes
  const size_t head = kScanHead, fbytes = flag_bytes(sh.tiles), sbytes = side_bytes<Op, T>(sh.tiles);
  void* scratch = nullptr;
  cudaError_t e = nt2cuda::stream_scratch(s, lookback_scratch<Op, T>(sh.tiles), &scratch, 1);
  if (e != cudaSuccess) return e;
  char* b = (char*)scratch;
  unsigned long long* ticket = (unsigned long long*)b;
  unsigned* err = (unsigned*)(b + 8);
  unsigned* flags = (unsigned*)(b + head);
  void* agg = b + head + fbytes;
  void* incl = b + head + fbytes + sbytes;
  if ((e = cudaMemsetAsync(b, 0, head + fbytes, s)) != cudaSuccess) return e;
  int vec = ((((uintptr_t)x | (uintptr_t)y) & 15u) == 0 && (rows * sizeof(T)) % 16 == 0) ? 1 : 0;
  auto k = one_pass ? k_scan_inner_1p<Op, T> : k_scan_inner<Op, T>;
  size_t grid = (size_t)sm_count() * (size_t)resident_blocks(k, 256);
  if (grid > sh.tiles) grid = sh.tiles;
  void* args[] = {(void*)&x, (void*)&y, (void*)&sh, (void*)&vec, (void*)&ticket, (void*)&flags, (void*)&agg,
                  (void*)&incl, (void*)&err};
  return launch_dependent(k, grid, 256, s, args);
}

static cudaError_t read_scan_wait_timeouts(unsigned long long* count)
{
  return cudaMemcpyFromSymbol(count, g_wait_timeouts, sizeof(unsigned long long));
}
static const timeout_reader_registration scan_wait_timeouts_reader(read_scan_wait_timeouts);

// Bounded waits that ran out since the library was loaded, over every kernel
// that counts them (scan look-backs, TMA fold barriers); synchronous.
inline cudaError_t wait_timeouts(unsigned long long* count) { return total_wait_timeouts(count); }

// A look-back wait that must run out: a two-tile column scanned with the
// ticket counter started at 1, so the block that takes tile 1 waits for a tile
// 0 that no block takes.  The kernel gives up after its bounded polls, writes
// NaN over tile 1 and sets the error word, which is returned in *failed.
inline cudaError_t selftest_wait_timeout(cudaStream_t s, unsigned* failed)
{
  using Op = fold::op_sum<true>;
  using K = scan_tiles<Op, float>;
  const size_t rows = 2 * K::TILE;
  float* buf = nullptr;
  char* scratch = nullptr;
  const size_t head = 256, fbytes = 256, sbytes = align256(2 * carry_bytes<Op, float>());
  cudaError_t e = cudaMalloc(&buf, rows * sizeof(float));
  if (e == cudaSuccess) e = cudaMalloc(&scratch, head + fbytes + 2 * sbytes);
  if (e == cudaSuccess) e = cudaMemsetAsync(buf, 0, rows * sizeof(float), s);
  if (e == cudaSuccess) e = cudaMemsetAsync(scratch, 0, head + fbytes, s);
  if (e == cudaSuccess) e = cudaMemsetAsync(scratch, 1, 1, s);    // ticket = 1
  if (e == cudaSuccess) {
    inner_shape sh;
    sh.rows = rows;
    sh.cols = 1;
    sh.tiles_per_col = 2;
    sh.tiles = 2;
    const float* x = buf;
    float* y = buf;
    int vec = 1;
    unsigned long long* ticket = (unsigned long long*)scratch;
    unsigned* err = (unsigned*)(scratch + 8);
    unsigned* flags = (unsigned*)(scratch + head);
    void* agg = scratch + head + fbytes;
    void* incl = scratch + head + fbytes + sbytes;
    void* args[] = {(void*)&x, (void*)&y, (void*)&sh, (void*)&vec, (void*)&ticket, (void*)&flags, (void*)&agg,
                    (void*)&incl, (void*)&err};
    e = launch_dependent(k_scan_inner<Op, float>, 2, 256, s, args);
    if (e == cudaSuccess) e = cudaMemcpyAsync(failed, err, sizeof(unsigned), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  }
  if (buf) cudaFree(buf);
  if (scratch) cudaFree(scratch);
  return e;
}

// The same for the streamed scan of x (which must be one it takes) into y.  kind 0:
// the tile at 0 is handed out to no block, so the gathers of the others run out;
// kind 1: no block waits for its own barriers at all.
inline cudaError_t selftest_stream_timeout(int kind, const float* x, float* y, size_t rows, size_t cols, cudaStream_t s,
                                           bool* ran_out)
{
  unsigned long long before = 0, after = 0;
  cudaError_t e = read_scan_wait_timeouts(&before);
  if (e == cudaSuccess)
    e = kind == 0 ? inner_scan_stream<true>(x, y, rows, cols, s, 1, tma::kMaxRounds, 1u << 10)
                  : inner_scan_stream<true>(x, y, rows, cols, s, 0, 0);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e == cudaSuccess) e = read_scan_wait_timeouts(&after);
  *ran_out = after > before;
  return e;
}

template <class Op, class T, int V>
cudaError_t outer_scan_v(const T* x, T* y, size_t rows, size_t cols, cudaStream_t s)
{
  using S = state_of<Op, T>;
  constexpr size_t ROWS = 256 * (size_t)V;
  outer_shape sh;
  sh.rows = rows;
  sh.cols = cols;
  sh.strips = (rows + ROWS - 1) / ROWS;
  // about two blocks per SM in all; a chunk is a whole number of 8-column groups
  const size_t want = (2 * (size_t)sm_count() + sh.strips - 1) / sh.strips;
  size_t cchunk = (cols + want - 1) / want;
  cchunk = (cchunk + 7) / 8 * 8;
  sh.cchunk = cchunk < 8 ? 8 : cchunk;
  sh.chunks = (cols + sh.cchunk - 1) / sh.cchunk;
  const size_t units = sh.strips * sh.chunks;
  S* totals = nullptr;
  cudaError_t e;
  if (sh.chunks > 1) {
    void* scratch = nullptr;
    if ((e = nt2cuda::stream_scratch(s, units * ROWS * sizeof(S), &scratch, 1)) != cudaSuccess) return e;
    totals = (S*)scratch;
    void* a1[] = {(void*)&x, (void*)&y, (void*)&sh, (void*)&totals};
    if ((e = launch_persistent(k_scan_outer<Op, T, V, false>, units * 256, 256, 2, s, a1)) != cudaSuccess)
      return e;
    void* a2[] = {(void*)&sh, (void*)&totals};
    if ((e = launch_persistent(k_scan_outer_prefix<Op, T, V>, sh.strips * ROWS, 256, 2, s, a2)) != cudaSuccess)
      return e;
  }
  void* a3[] = {(void*)&x, (void*)&y, (void*)&sh, (void*)&totals};
  return launch_persistent(k_scan_outer<Op, T, V, true>, units * 256, 256, 2, s, a3);
}

// The TMA-staged row scan (k_scan_outer_tma): one block per strip of
// 128 bytes of rows walking all columns.  cudaErrorNotSupported, before
// anything is launched, when the tensor maps cannot be made.
template <class Op, class T>
cudaError_t outer_scan_staged(const T* x, T* y, size_t rows, size_t cols, cudaStream_t s)
{
  constexpr int BR = outer_tma_rows<T>(), BC = kOuterTmaCols, STAGES = 6;
  PFN_cuTensorMapEncodeTiled_v12000 encode = tma::tensor_map_encoder();
  if (!encode) return cudaErrorNotSupported;
  CUtensorMap xmap, ymap;
  const cuuint64_t gdim[2] = {(cuuint64_t)rows, (cuuint64_t)cols};
  const cuuint64_t gstride[1] = {(cuuint64_t)(rows * sizeof(T))};
  const cuuint32_t box[2] = {(cuuint32_t)BR, (cuuint32_t)BC};
  const cuuint32_t estride[2] = {1, 1};
  const CUtensorMapDataType dt = sizeof(T) == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT64;
  if (encode(&xmap, dt, 2, (void*)x, gdim, gstride, box, estride, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS ||
      encode(&ymap, dt, 2, (void*)y, gdim, gstride, box, estride, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return cudaErrorNotSupported;
  outer_tma_shape sh;
  sh.rows = rows;
  sh.cols = cols;
  sh.strips = (rows + BR - 1) / BR;
  sh.ctiles = (cols + BC - 1) / BC;
  sh.wait_rounds = tma::kMaxRounds;
  auto k = k_scan_outer_tma<Op, T, STAGES>;
  const int smem = STAGES * BR * BC * (int)sizeof(T);
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  void* args[] = {(void*)&xmap, (void*)&ymap, (void*)&sh};
  return launch_dependent(k, sh.strips, 256, s, args, smem);
}

template <class Op, class T>
cudaError_t outer_scan(const T* x, T* y, size_t rows, size_t cols, cudaStream_t s)
{
  if (!rows || !cols) return cudaSuccess;
  constexpr int V = 16 / (int)sizeof(T);
  // at least one strip of 128 bytes of rows per SM: the staged single pass
  if ((((uintptr_t)x | (uintptr_t)y) & 15u) == 0 && rows % V == 0 && rows < ((size_t)1 << 31) &&
      cols < ((size_t)1 << 31) && rows / (size_t)outer_tma_rows<T>() >= (size_t)sm_count()) {
    const cudaError_t e = outer_scan_staged<Op, T>(x, y, rows, cols, s);
    if (e != cudaErrorNotSupported) return e;
  }
  if ((((uintptr_t)x | (uintptr_t)y) & 15u) == 0 && rows % V == 0) return outer_scan_v<Op, T, V>(x, y, rows, cols, s);
  return outer_scan_v<Op, T, 1>(x, y, rows, cols, s);
}

template <class Op, class T>
cudaError_t scan_dim(const T* x, T* y, size_t rows, size_t cols, int dim, cudaStream_t s)
{
  return dim == 1 ? inner_scan<Op, T>(x, y, rows, cols, s) : outer_scan<Op, T>(x, y, rows, cols, s);
}

}  // namespace scan
}  // namespace nt2cuda
