// tcgen05.cuh -- shared helpers for the kernels on the 5th-generation tensor
// cores (sm_100a): shared-memory matrix descriptors, tcgen05.mma / commit /
// ld, the TMEM fences, tiled TMA loads (no multicast) and the driver's tensor
// map encoder.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <mutex>

#include "common.cuh"

namespace lc {

// K-major operand, 128-byte swizzle: 8-row groups of 1024 bytes (SBO), start
// address advanced by 32 bytes per K step inside the swizzle atom.
LC_D uint64_t umma_desc_sw128(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFF);  // start address
  d |= (uint64_t)1 << 16;                   // leading byte offset (unused here)
  d |= (uint64_t)(1024 >> 4) << 32;         // stride byte offset
  d |= (uint64_t)1 << 46;                   // descriptor version
  d |= (uint64_t)2 << 61;                   // layout: 128-byte swizzle
  return d;
}

// K-major operand without swizzle: 8-row x 16-byte core matrices, `lbo`
// bytes to the next one along K, `sbo` bytes to the next 8-row group.
LC_D uint64_t umma_desc_noswz(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFF);
  d |= (uint64_t)((lbo >> 4) & 0x3FFF) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3FFF) << 32;
  d |= (uint64_t)1 << 46;  // descriptor version; layout 0: no swizzle
  return d;
}

// Acquire of a tensor map that lies in global memory and was copied there from
// the host: without it the thread's TMA loads may use a descriptor cached from an
// earlier map at the same address (its box, and so the bytes that arrive, may differ).
LC_D void tensormap_acquire(const CUtensorMap* map) {
  asm volatile("fence.proxy.tensormap::generic.acquire.sys [%0], 128;" ::"l"(map) : "memory");
}

LC_D void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
          smem_u32(dst)),
      "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar))
      : "memory");
}

LC_D void mma_i8(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate));
}

LC_D void mma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   smem_u32(bar))
               : "memory");
}

LC_D void tmem_ld16(uint32_t addr, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
        "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]),
        "=r"(v[15])
      : "r"(addr));
}

LC_D void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
LC_D void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// K-major operand, 64-byte swizzle: 64-byte rows, 8-row groups of 512 bytes
// (SBO), start address advanced by 32 bytes per K step inside the atom.
LC_D uint64_t umma_desc_sw64(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFF);  // start address
  d |= (uint64_t)1 << 16;                   // leading byte offset (unused here)
  d |= (uint64_t)(512 >> 4) << 32;          // stride byte offset
  d |= (uint64_t)1 << 46;                   // descriptor version
  d |= (uint64_t)4 << 61;                   // layout: 64-byte swizzle
  return d;
}

LC_D void tmem_ld8(uint32_t addr, uint32_t (&v)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
               : "r"(addr));
}

LC_D void tmem_ld4(uint32_t addr, uint32_t (&v)[4]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3])
               : "r"(addr));
}

LC_D void tma_load_3d(void* dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
          smem_u32(dst)),
      "l"(map), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
      : "memory");
}

// MN-major operand: LBO = bytes to the next atom along M/N, SBO = bytes to
// the next 8-row group along K; layout 2 = 128-byte swizzle, 4 = 64-byte,
// 6 = 32-byte.
LC_D uint64_t umma_desc_mn(uint32_t saddr, uint32_t lbo, uint32_t sbo, uint32_t layout) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFF);
  d |= (uint64_t)((lbo >> 4) & 0x3FFF) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3FFF) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)layout << 61;
  return d;
}

// 16-byte global -> shared copy of `bytes` (0..16) source bytes, the rest
// zero (src and dst 16-byte aligned; no byte is read when bytes = 0), and the
// per-thread commit / wait of those copies.
LC_D void cp_async16_zfill(uint32_t dst, const void* src, uint32_t bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
LC_D void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
LC_D void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Eight outputs sum_l 2^(8l) D_l mod p (p = 2^64 - 2^32 + 1, |D_l| <= 256 * 128 *
// 255, so D_l + 2^8 D_(l+1) fits int32), each as a 64-bit value congruent mod p
// but not necessarily canonical: every reader of the witness transforms -- the
// byte-limb slot products and the 160-bit integer products -- takes any 64-bit
// representative.  A = D0 + 2^8 D1 + 2^16 D2 + 2^24 D3 and B (limbs 4..7) are
// exact in int64 (below 2^47.1).  With hB:lB = B (hB signed) and X = A - hB,
//   A + 2^32 B == X + 2^32 (hB + lB)   (2^64 == 2^32 - 1),
// so the low word is X's and the high word s + lB with s = hi(X) + hB, |s| < 2^17.
// That sum leaves [0, 2^32) by k = 1 or -1 only when its low word lies within
// 2^18 of the ends (2^-13 of the outputs); then k (2^32 - 1) is added, which
// stays inside [0, 2^64).  Zeros (zero ring elements, the columns past the batch)
// lie there too and need nothing, which the top bits of lB and of the low word
// tell: they differ for every sum that passes an end.  Correcting zeros with the
// rest took tc_ntt_kernel a fifth longer; asking for the top bits at once 1 % (852
// -> 861 us at 128 witnesses of 2^16 ring elements).
LC_D void gl_fold_limbs8(const uint32_t (&d)[8][8], uint64_t (&out)[8]) {
  uint32_t hi[8], lo[8];
  int32_t s[8];
  bool edge = false;
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    const int32_t p01 = (int32_t)d[0][u] + (int32_t)d[1][u] * 256;
    const int32_t p23 = (int32_t)d[2][u] + (int32_t)d[3][u] * 256;
    const int32_t p45 = (int32_t)d[4][u] + (int32_t)d[5][u] * 256;
    const int32_t p67 = (int32_t)d[6][u] + (int32_t)d[7][u] * 256;
    const int64_t A = (int64_t)p23 * 65536 + p01;
    const int64_t B = (int64_t)p67 * 65536 + p45;
    const int32_t hB = (int32_t)(B >> 32);
    const int64_t X = A - hB;
    s[u] = (int32_t)(X >> 32) + hB;
    lo[u] = (uint32_t)X;
    hi[u] = (uint32_t)B + (uint32_t)s[u];
    edge |= hi[u] + 0x40000u < 0x80000u;
  }
#pragma unroll
  for (int u = 0; u < 8; ++u) out[u] = (uint64_t)hi[u] << 32 | lo[u];
  if (edge) {
    uint32_t passed = 0;
#pragma unroll
    for (int u = 0; u < 8; ++u) passed |= hi[u] ^ (hi[u] - (uint32_t)s[u]);
    if ((int32_t)passed >= 0) return;
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int k = s[u] >= 0 ? (int)(hi[u] < (uint32_t)s[u]) : -(int)(hi[u] >= (uint32_t)s[u]);
      out[u] += (uint64_t)(int64_t)k * 0xFFFFFFFFull;
    }
  }
}

// ------------------------------------------------------------------ host side

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(ptr);
    cudaGetLastError();
  });
  return fn;
}


}  // namespace lc
