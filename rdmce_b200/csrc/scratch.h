// scratch.h -- device buffers that outlive a call (host declarations).
#pragma once
#include <cuda_runtime.h>

#include <cstddef>

#include "internal.h"

namespace mce {

// Device scratch owned by one solver context: buffers keyed by purpose, grown
// on demand and kept for reuse (the role of the reference's BufferManager,
// include/context_gpu.cuh:4-32, without its worst-case sizing).
struct Scratch {
  static constexpr int kSlots = 8;
  int device = 0;
  // set: buffers are allocated and freed stream-ordered on this stream (no
  // device-wide synchronisation when one grows), for an owner whose work
  // stays on that stream (a server dispatcher)
  cudaStream_t ordered = nullptr;
  void *ptr[kSlots] = {};
  size_t bytes[kSlots] = {};
  size_t most[kSlots] = {};  // larger requests are turned down as if memory had run out (0: no limit)
  void *get(int purpose, size_t n, mce_status *st);
  void release();
  ~Scratch() { release(); }
};
// the default per-device context used by single-graph calls, and its lock
Scratch *default_scratch(int device);
void lock_default(int device);
void unlock_default(int device);

}  // namespace mce
