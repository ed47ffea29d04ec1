// nt2cuda/scratch.cuh -- per-stream device scratch for multi-block kernels.
//
// The folds keep per-block partials and arrival counters in global memory.
// Each (stream, device, slot) gets its own buffer, so kernels enqueued on
// different streams never share scratch; calls on one stream are ordered and
// reuse it.  A buffer only grows; growing synchronises its stream first.  The
// first call on a stream allocates (cudaMalloc), so make it before capturing
// that stream into a CUDA graph.  A graph keeps the addresses, so its launches
// have to be ordered with the calls and graphs that share them (captured folds
// of columns of up to 4096 16-byte groups use none), and a buffer that a larger
// one replaces stays allocated: the larger one is at least twice its size, so
// those before the last take less than it together.  The folds' arrival
// counters have a slot of their own: they start at zero (a buffer is cleared
// when allocated), every fold leaves the ones it used at zero, and nothing else
// is written there -- partials, which other kernels overwrite freely, live in
// another slot.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <mutex>
#include <unordered_map>

namespace nt2cuda {

struct scratch_pool {
  struct entry { void* p = nullptr; size_t bytes = 0; };
  std::mutex m;
  std::unordered_map<uintptr_t, entry> by_key;
  unsigned long long allocations = 0;     // cudaMalloc calls made for scratch so far
};
inline scratch_pool& global_scratch_pool() { static scratch_pool p; return p; }

// slot 0: fold arrival counters only; slot 1: per-call data (batched-launch
// descriptors, scan flags and carries); slot 2: fold partials; slot 3
// (kResultSlot): device results the C++ front end reads back (globalsum).
constexpr int kResultSlot = 3;
inline cudaError_t stream_scratch(cudaStream_t s, size_t bytes, void** out, int slot = 0, size_t room = 0);

// The two buffers of a fold of n outputs, each cut into `splits` segments: a
// zero-valued arrival counter and splits * states partial states of `partial_bytes`
// for each output (none where it is not cut).  Outside capture they are made large
// enough for `wide` segments too, the cut of a captured call.
inline cudaError_t fold_scratch(cudaStream_t s, size_t n, size_t splits, size_t wide, size_t partial_bytes,
                                unsigned** counters, void** partials, size_t states = 1)
{
  const size_t most = splits > wide ? splits : wide;
  void* c = nullptr;
  *counters = nullptr;
  *partials = nullptr;
  if (most <= 1) return cudaSuccess;
  cudaError_t e = stream_scratch(s, splits > 1 ? n * sizeof(unsigned) : 0, &c, 0, n * sizeof(unsigned));
  if (e != cudaSuccess) return e;
  e = stream_scratch(s, splits > 1 ? n * splits * states * partial_bytes : 0, partials, 2, n * most * states * partial_bytes);
  *counters = (unsigned*)c;
  return e;
}

inline uintptr_t scratch_key(cudaStream_t s, int slot)
{
  int dev = 0;
  cudaGetDevice(&dev);
  return (reinterpret_cast<uintptr_t>(s) * 64u + (uintptr_t)dev) * 4u + (uintptr_t)slot;
}

// Whether the stream is being captured into a CUDA graph.
inline bool capturing(cudaStream_t s)
{
  cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &st) == cudaSuccess) return st != cudaStreamCaptureStatusNone;
  (void)cudaGetLastError();
  return false;
}

// At least `bytes`; a buffer that grows, and outside capture one smaller than
// `room`, becomes the larger of the two.
inline cudaError_t stream_scratch(cudaStream_t s, size_t bytes, void** out, int slot, size_t room)
{
  const uintptr_t key = scratch_key(s, slot);
  scratch_pool& P = global_scratch_pool();
  std::lock_guard<std::mutex> g(P.m);
  scratch_pool::entry& e = P.by_key[key];
  if (room < bytes) room = bytes;
  if (e.bytes < room && (e.bytes < bytes || !capturing(s))) {
    cudaError_t err = e.p ? cudaStreamSynchronize(s) : cudaSuccess;   // (an error under capture)
    if (err != cudaSuccess) return err;
    size_t want = room < 4096 ? 4096 : room;
    if (want < 2 * e.bytes) want = 2 * e.bytes;
    void* p = nullptr;
    if ((err = cudaMalloc(&p, want)) != cudaSuccess) return err;
    ++P.allocations;
    if ((err = cudaMemsetAsync(p, 0, want, s)) != cudaSuccess) {
      cudaFree(p);
      return err;
    }
    e.p = p;
    e.bytes = want;
  }
  *out = e.p;
  return cudaSuccess;
}

}  // namespace nt2cuda
