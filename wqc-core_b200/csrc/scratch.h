// Device memory of the reads (environments of Pauli sums and shots), kept
// between calls: a cudaMalloc and a cudaFree a call cost more than most reads
// do.  One pool a device for all its states, contexts and threads, of at most
// kScratchKeep idle bytes.  A block belongs to one call at a time and comes
// back once the stream that used it has drained.  Idle blocks are given up when
// an allocation of this library fails, when the last state of the device is
// destroyed, when the free memory is asked for, and when the context is closed.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

namespace wqc {

constexpr size_t kScratchKeep = size_t(512) << 20;

// An idle block of at least `bytes` (its size in *cap), the smallest there is,
// or nullptr.
void* scratch_take(int device, size_t bytes, size_t* cap);
// Back to the pool, or freed if it alone is more than the pool keeps.
void scratch_give(int device, void* p, size_t cap);
// Frees the idle blocks; true if there were any.
bool scratch_release(int device);
// A state of the device was created (+1) or destroyed (-1).
void scratch_states(int device, int change);

// cudaMalloc on the current device, once more without the idle blocks.
cudaError_t device_malloc(void** p, size_t bytes);
// Whether `need` bytes are free on the current device, idle blocks given up if
// it takes them; the free bytes in *free_bytes.
cudaError_t device_room(uint64_t need, size_t* free_bytes);

}  // namespace wqc
