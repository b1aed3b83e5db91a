// blocks.cu -- device blocks of keys and of their scratch.
//
// Making a key costs a cudaMalloc and destroying it a cudaFree, each a driver
// call of 100 us and more that also serialises with the device's other work; a
// verifier that derives its key from the seed on every call paid both several
// times per call (from_seed + one commit, k = 2, m = 2000: 940 us).
// Freed blocks of up to 32 MiB are kept for the next key, at most 64 MiB per
// device, the newest; they go back to the driver when an allocation of this library fails
// and when the last plan and key of the process is destroyed.
//
// A key may be destroyed while its commits still run, on any stream.  Its block
// is handed out again only after a synchronisation of the device, and that is
// left to the next key's creation (block_settle): a synchronisation while some
// stream captures a graph ends the capture, and a key can go at any time (a
// garbage collector), while creating one never was possible there.
#include "blocks.h"

#include <cuda_runtime.h>

#include <mutex>
#include <vector>

#include "../../include/lattice_cuda.h"

namespace lc {

constexpr size_t kBlockKeepMax = (size_t)32 << 20, kBlockKeepTotal = (size_t)64 << 20;

struct KeptBlock {
  void* p;
  size_t bytes;
  int device;
  bool idle;  // no queued work uses it
};
static std::mutex g_block_mu;
static std::vector<KeptBlock> g_blocks;
static long g_block_users = 0;

static size_t block_size(size_t bytes) {  // what may be kept has at most 1/8 unused
  if (bytes > kBlockKeepMax) return bytes;
  size_t step = 512;
  while (step * 16 < bytes) step *= 2;
  return (bytes + step - 1) / step * step;
}

// frees the kept blocks (of every device); g_block_mu held
static void block_drain() {
  for (const KeptBlock& b : g_blocks) cudaFree(b.p);
  g_blocks.clear();
}

cudaError_t dev_malloc(void** p, size_t bytes) {
  cudaError_t e = cudaMalloc(p, bytes);
  if (e != cudaErrorMemoryAllocation) return e;
  std::lock_guard<std::mutex> lk(g_block_mu);
  if (g_blocks.empty()) return e;
  cudaGetLastError();
  block_drain();
  return cudaMalloc(p, bytes);
}

int block_alloc(void** p, size_t bytes) {
  const size_t size = block_size(bytes);
  int dev = 0;
  *p = nullptr;
  if (cudaGetDevice(&dev) != cudaSuccess) {
    cudaGetLastError();
    return LC_ERR_CUDA;
  }
  {
    std::lock_guard<std::mutex> lk(g_block_mu);
    for (size_t i = 0; i < g_blocks.size(); ++i)
      if (g_blocks[i].bytes == size && g_blocks[i].device == dev && g_blocks[i].idle) {
        *p = g_blocks[i].p;
        g_blocks.erase(g_blocks.begin() + (long)i);
        return LC_OK;
      }
  }
  if (dev_malloc(p, size) == cudaSuccess) return LC_OK;
  cudaGetLastError();
  *p = nullptr;
  return LC_ERR_OUT_OF_MEMORY;
}

void block_free(void* p, size_t bytes, int device, bool idle) {
  if (!p) return;
  const size_t size = block_size(bytes);
  if (size > kBlockKeepMax) {
    cudaFree(p);
    return;
  }
  std::lock_guard<std::mutex> lk(g_block_mu);
  g_blocks.push_back({p, size, device, idle});
  size_t kept = 0;
  for (const KeptBlock& b : g_blocks)
    if (b.device == device) kept += b.bytes;
  // the oldest make room: a list full of sizes that no key asks for any more would
  // leave every later key to the driver
  for (size_t i = 0; kept > kBlockKeepTotal;) {
    if (g_blocks[i].device != device) {
      ++i;
      continue;
    }
    kept -= g_blocks[i].bytes;
    cudaFree(g_blocks[i].p);
    g_blocks.erase(g_blocks.begin() + (long)i);
  }
}

int block_grow(void** p, size_t* have, size_t need) {
  if (need <= *have) return LC_OK;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) {
    cudaGetLastError();
    return LC_ERR_CUDA;
  }
  block_free(*p, *have, dev, false);  // queued work may use it
  *p = nullptr;
  *have = 0;
  const int rc = block_alloc(p, need);
  if (!rc) *have = need;
  return rc;
}

void block_settle() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) {
    cudaGetLastError();
    return;
  }
  std::lock_guard<std::mutex> lk(g_block_mu);
  bool any = false;
  for (const KeptBlock& b : g_blocks) any |= b.device == dev && !b.idle;
  if (!any) return;
  if (cudaDeviceSynchronize() != cudaSuccess) {  // they stay as they are
    cudaGetLastError();
    return;
  }
  for (KeptBlock& b : g_blocks) b.idle |= b.device == dev;
}

void block_users(int delta) {
  std::lock_guard<std::mutex> lk(g_block_mu);
  g_block_users += delta;
  if (g_block_users == 0) block_drain();
}

}  // namespace lc
