"""The kept device blocks of keys (lzx_b200/csrc/blocks.cu) against a fake CUDA runtime, on the CPU.

The source is compiled with the host compiler against a stand-in
``cuda_runtime.h`` whose allocator hands out numbers, counts the driver calls
and fails on request.
"""
import os
import subprocess

import pytest

from conftest import ROOT

RUNTIME = r"""
#pragma once
#include <stddef.h>
enum cudaError_t { cudaSuccess = 0, cudaErrorMemoryAllocation = 2, cudaErrorOther = 900 };
struct Fake {
  long mallocs = 0, frees = 0, syncs = 0;
  int device = 0;
  size_t live = 0, limit = (size_t)1 << 40;
  bool sync_fails = false;
};
extern Fake fake;
cudaError_t cudaMalloc(void** p, size_t bytes);
cudaError_t cudaFree(void* p);
cudaError_t cudaGetDevice(int* d);
cudaError_t cudaGetLastError();
cudaError_t cudaDeviceSynchronize();
"""

FAKE = r"""
#include <cuda_runtime.h>
#include <cstdio>
#include <cstdlib>
#include <map>
#include <vector>
#include "blocks.h"
#include "lattice_cuda.h"
Fake fake;
static std::map<void*, size_t> sizes;
static char* next_p = reinterpret_cast<char*>(4096);
cudaError_t cudaMalloc(void** p, size_t bytes) {
  ++fake.mallocs;
  if (fake.live + bytes > fake.limit) return cudaErrorMemoryAllocation;
  *p = next_p;
  next_p += (bytes + 511) / 512 * 512;
  sizes[*p] = bytes;
  fake.live += bytes;
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  ++fake.frees;
  fake.live -= sizes.at(p);  // throws for a block that is not there
  sizes.erase(p);
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) { *d = fake.device; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { ++fake.syncs; return fake.sync_fails ? cudaErrorOther : cudaSuccess; }
#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); std::exit(1); } } while (0)
using namespace lc;
constexpr size_t MiB = 1 << 20;
int main() {
  block_users(1);
  BODY
  block_users(-1);
  CHECK(fake.live == 0 && sizes.empty());
  return 0;
}
"""


def run(tmp_path, body):
    (tmp_path / "cuda_runtime.h").write_text(RUNTIME)
    (tmp_path / "main.cpp").write_text(FAKE.replace("BODY", body))
    src = os.path.join(ROOT, "lzx_b200", "csrc")
    exe = str(tmp_path / "blocks")
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", str(tmp_path), "-I", src,
                    "-I", os.path.join(ROOT, "include"), "-o", exe, str(tmp_path / "main.cpp"),
                    "-x", "c++", os.path.join(src, "blocks.cu")], check=True, capture_output=True, text=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr


BODIES = {
    # a block that queued work may use is not synchronised for when it is freed, nor
    # handed out before the device was synchronised
    "busy": """
  void *a, *b, *c;
  CHECK(block_alloc(&a, MiB) == LC_OK);
  block_free(a, MiB, 0, false);
  CHECK(fake.syncs == 0);
  CHECK(block_alloc(&b, MiB) == LC_OK && b != a && fake.mallocs == 2 && fake.syncs == 0);
  block_settle();
  CHECK(fake.syncs == 1);
  block_settle();
  CHECK(fake.syncs == 1);
  CHECK(block_alloc(&c, MiB) == LC_OK && c == a && fake.mallocs == 2);
  block_free(b, MiB, 0, true);
  CHECK(block_alloc(&b, MiB) == LC_OK && fake.mallocs == 2 && fake.syncs == 1);
  block_free(b, MiB, 0, true);
  block_free(c, MiB, 0, true);""",
    # a failed synchronisation hands nothing out; another device's blocks stay as they are
    "device": """
  void *a, *b;
  CHECK(block_alloc(&a, MiB) == LC_OK);
  block_free(a, MiB, 0, false);
  fake.sync_fails = true;
  block_settle();
  CHECK(block_alloc(&b, MiB) == LC_OK && b != a);
  block_free(b, MiB, 0, true);
  fake.sync_fails = false;
  fake.device = 1;
  block_settle();
  CHECK(fake.syncs == 1);
  CHECK(block_alloc(&b, MiB) == LC_OK && fake.mallocs == 3);
  block_free(b, MiB, 1, true);""",
    # a full list makes room: the oldest blocks go back, the newest are there for the next key
    "evict": """
  void *a[5], *b;
  for (int i = 0; i < 5; ++i) CHECK(block_alloc(&a[i], (16 + 2 * i) * MiB) == LC_OK);
  for (int i = 0; i < 5; ++i) block_free(a[i], (16 + 2 * i) * MiB, 0, true);  // 100 MiB, of which 64 are kept
  CHECK(fake.frees == 3 && fake.live == 46 * MiB);
  CHECK(block_alloc(&b, 24 * MiB) == LC_OK && b == a[4] && fake.mallocs == 5);
  block_free(b, 24 * MiB, 0, true);
  CHECK(block_alloc(&b, 16 * MiB) == LC_OK && fake.mallocs == 6);
  block_free(b, 16 * MiB, 0, true);
  CHECK(block_alloc(&b, 40 * MiB) == LC_OK);  // too large to keep: the list stays
  long frees = fake.frees;
  block_free(b, 40 * MiB, 0, true);
  CHECK(fake.frees == frees + 1);""",
    # an allocation that the driver refuses takes the kept blocks back first
    "drain": """
  void *a, *b;
  int* c = nullptr;
  CHECK(block_alloc(&a, 30 * MiB) == LC_OK && block_alloc(&b, 30 * MiB) == LC_OK);
  block_free(a, 30 * MiB, 0, true);
  block_free(b, 30 * MiB, 0, false);
  fake.limit = 64 * MiB;
  CHECK(dev_malloc(&c, 40 * MiB) == cudaSuccess && c && fake.live == 40 * MiB && fake.frees == 2);
  void* d;
  CHECK(dev_malloc(&d, 40 * MiB) == cudaErrorMemoryAllocation && fake.frees == 2);
  CHECK(block_alloc(&d, 40 * MiB) == LC_ERR_OUT_OF_MEMORY && d == nullptr);
  cudaFree(c);""",
    # the scratch of a key goes to the next one, after a synchronisation
    "scratch": """
  void *a = nullptr, *b = nullptr;
  size_t have_a = 0, have_b = 0;
  CHECK(block_grow(&a, &have_a, 3 * MiB) == LC_OK && have_a == 3 * MiB);
  void* was = a;
  CHECK(block_grow(&a, &have_a, 2 * MiB) == LC_OK && a == was && have_a == 3 * MiB);
  CHECK(block_grow(&a, &have_a, 5 * MiB) == LC_OK && a != was && have_a == 5 * MiB && fake.frees == 0 && fake.syncs == 0);
  CHECK(block_grow(&b, &have_b, 3 * MiB) == LC_OK && b != was && fake.mallocs == 3);
  block_free(b, have_b, 0, false);
  block_settle();
  b = nullptr;
  have_b = 0;
  CHECK(block_grow(&b, &have_b, 3 * MiB) == LC_OK && fake.mallocs == 3);
  fake.limit = 8 * MiB;
  CHECK(block_grow(&b, &have_b, 20 * MiB) == LC_ERR_OUT_OF_MEMORY && !b && have_b == 0);
  block_free(a, have_a, 0, true);""",
}


def test_every_allocation_can_take_the_kept_blocks_back():
    src = os.path.join(ROOT, "lzx_b200", "csrc")
    for f in sorted(os.listdir(src)):
        if f != "blocks.cu":
            with open(os.path.join(src, f)) as fh:
                assert "cudaMalloc(" not in fh.read(), f


@pytest.mark.parametrize("name", list(BODIES))
def test_blocks(tmp_path, name):
    run(tmp_path, BODIES[name])
