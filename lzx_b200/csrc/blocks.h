// blocks.h -- device memory of keys: freed blocks are kept for the next key.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>

namespace lc {

// cudaMalloc for everything this library allocates: when the driver has no more, the
// kept blocks go back to it first.
cudaError_t dev_malloc(void** p, size_t bytes);
template <class T>
cudaError_t dev_malloc(T** p, size_t bytes) {
  return dev_malloc(reinterpret_cast<void**>(p), bytes);
}

// block_alloc hands out a kept block of the same (rounded) size that no queued
// work uses, or driver memory.  `idle` tells block_free that nothing queued uses
// the block any more; the others wait in the list for block_settle, which
// synchronises the current device when it has such blocks (for calls that are
// synchronous anyway).
int block_alloc(void** p, size_t bytes);
void block_free(void* p, size_t bytes, int device, bool idle);
void block_settle();
// A key's scratch: a block of at least `need` bytes in *p (its size in *have); a
// smaller one there is freed.
int block_grow(void** p, size_t* have, size_t need);
void block_users(int delta);  // live plans and keys: the last one frees what is kept

}  // namespace lc
