// gl_ntt.cu -- batched Goldilocks NTT / INTT on the INT8 tensor cores
// (tcgen05.mma .kind::i8, sm_100a), exact.
//
// The transforms of NttTables::forward_fast / inverse_fast
// (lattice-ring/src/ntt.rs:118-146, 187-216) over p = 2^64 - 2^32 + 1 for
// n = N1 N2 = 64 .. 1024, as two small dense transforms with one general
// product per value between them:
//   out[x1 + N1 x2] = sum_y2 VB[x2][y2] W[y2][x1] sum_y1 VA[x1][y1] in[N2 y1 + y2]
//   forward (psi of order 2n, omega = psi^2):
//     VA[x1][y1] = psi^(N2 y1 (2 x1 + 1)), W[y2][x1] = psi^(y2 (2 x1 + 1)),
//     VB[x2][y2] = omega^(N1 x2 y2)
//   inverse:
//     VA[x1][y1] = omega^(-N2 x1 y1), W[y2][x1] = omega^(-x1 y2) psi^(-x1) / n,
//     VB[x2][y2] = omega^(-N1 x2 y2) psi^(-N1 x2)
// A dense N-point transform of 64-bit residues is an exact byte GEMM: the value
// bytes b_(y,lw) are the A operand as they lie in memory, and with the byte
// limbs V_l of V[x][y] 2^(8 lw) mod p
//   D_l[x] = sum_(y,lw) b_(y,lw) V_l[x][(y,lw)]   (u8 x u8 -> s32, K = 8N <= 256,
// at most 256 * 255^2, so D_l + 2^8 D_(l+1) fits 32 bits), and the result is
// sum_l 2^(8l) D_l mod p (gl_fold_bytes4).
//
// A CTA (one per SM, persistent) takes tiles of 4096 values = 4096 / n
// polynomials: pass A has 4096 / N1 rows (poly, y2), pass B 4096 / N2 rows
// (poly, x1), both 128-row M blocks of 8N columns (limb, x) that fill 256 TMEM
// columns.  Warps 0-15 fold pass A, multiply by W and write pass B's operand to
// shared memory; warps 16-23 fold pass B and store it (lanes along x1:
// contiguous); 24-27 load the tile (two LDG.64, one STS.128 per pair of y1);
// 28 issues the MMAs, A of the next tile before B of this one.  Folding warps
// take four columns x at a time, which fits 64 registers.  All waits are
// bounded.
//
// Bound: the integer instructions of the two folds and the product between
// them, about 100 per value with the loads and stores whatever n is, where the
// register transform (ntt_tile_kernel) issues 54 per butterfly, 0.5 log2 n
// butterflies per value.  30 011 inverse transforms of n = 1024: 499 -> 170 us
// (189 with eight warps per fold), 75 us for the bytes; 2^25 values of n = 64
// 256 -> 167, n = 256 400 -> 169, n = 512 399 -> 186 us.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <mutex>

#include "../../include/lattice_cuda.h"
#include "arith.cuh"
#include "common.cuh"
#include "internal.h"
#include "tcgen05.cuh"

namespace lc {

constexpr int kGnTile = 4096;  // values per tile
constexpr int kGnFold1 = 16, kGnFold2 = 8, kGnLoad = 4;  // warps folding pass A and pass B, loader warps
constexpr int kGnThreads = 32 * (kGnFold1 + kGnFold2 + kGnLoad + 1);

// WIT: the commitment's witness transform -- polynomials (j, b), b fastest, read
// from w[b][j][n] and written to What_T[t][j][b_pad], zeros in the columns from
// batch on.  Pass B's rows then run along the polynomials, so that a warp's
// lanes store a run of one slot.  The register form does the butterflies of the
// padding too and is bound by its multiplications: whole commitments of kappa =
// 4 went from 1177 to 970 us (d = 128, m = 8192, 128 witnesses), from 120 to 110
// (d = 128, m = 3001, 20) and from 1289 to 1096 (d = 256, m = 4096, 128).  Not
// taken, as they were slower or no faster: d = 64 (952 us against 950 at m =
// 16384, 73 against 77 at m = 4096 and 20 witnesses) and byte digits, which this
// loader reads one by one (1131 us against 1293 at d = 128).
template <int LOG_N1, int LOG_N2, bool WIT>
struct GnCfg {
  static constexpr int N1 = 1 << LOG_N1, N2 = 1 << LOG_N2, N = N1 * N2;
  static constexpr int P = kGnTile / N;  // polynomials per tile
  static constexpr int RA = kGnTile / N1, RB = kGnTile / N2;  // rows of the passes
  // operand: 16-byte K chunk c (two values) of row r at c * LB + 16 r; the pad per
  // column of chunks spreads a warp's stores of pass B's operand over the banks
  static constexpr int LBA = RA * 16 + 16, LBB = RB * 16 + (WIT ? 16 * (32 / N2) : 16);
  static constexpr int VA = 64 * N1 * N1, VB = 64 * N2 * N2;  // (8N)^2 bytes
  static constexpr int OFF_VB = VA, OFF_W = OFF_VB + VB, OFF_A = OFF_W + 8 * N;
  static constexpr int OFF_B = OFF_A + N1 / 2 * LBA, OFF_BAR = OFF_B + N2 / 2 * LBB;
  static constexpr size_t SMEM = 128 + OFF_BAR + 128;
  static constexpr int TABLE = OFF_A;  // device table: VA, VB, W in shared-memory order
  static_assert(N1 >= 8 && N1 <= 32 && N2 >= 8 && N2 <= 32, "passes");
  static_assert(OFF_BAR % 8 == 0 && SMEM <= 227 * 1024, "shared memory");
};

// D = s32, A = B = u8, both K-major, M = 128, N = 8 * points
LC_HD constexpr uint32_t gn_idesc(int points) {
  return (2u << 4) | ((uint32_t)points << 17) | ((128u >> 4) << 24);
}

struct GnParams {
  const uint64_t* in;
  uint64_t* out;
  const uint4* table;
  unsigned long long count;  // polynomials
  uint32_t tiles;
  uint32_t* err;
  uint32_t m, batch, b_pad;  // witness transforms
};

// Four values sum_l 2^(8l) D_l mod p, 0 <= D_l <= 256 * 255^2, as any 64-bit
// representative: gl_fold_limbs8 without signs -- the high word's s is not
// negative, so the only wrap is a carry.
LC_D void gl_fold_bytes4(const uint32_t (&d)[8][4], uint64_t (&out)[4]) {
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const uint32_t p01 = d[0][u] + d[1][u] * 256, p23 = d[2][u] + d[3][u] * 256;
    const uint32_t p45 = d[4][u] + d[5][u] * 256, p67 = d[6][u] + d[7][u] * 256;
    const uint64_t A = (uint64_t)p23 * 65536 + p01, B = (uint64_t)p67 * 65536 + p45;
    const uint32_t hB = (uint32_t)(B >> 32);
    const uint64_t X = A - hB;
    const uint32_t s = (uint32_t)(X >> 32) + hB;  // below 2^18; X < 0 only when hB > 0
    const uint32_t hi = (uint32_t)B + s;
    out[u] = (uint64_t)hi << 32 | (uint32_t)X;
    if (hi < s) out[u] += kGlEps;  // 2^64 == 2^32 - 1; the sum is below 2^50
  }
}

template <int LOG_N1, int LOG_N2, bool WIT>
__global__ void __launch_bounds__(kGnThreads, 1) gl_ntt_kernel(const __grid_constant__ GnParams p) {
  using C = GnCfg<LOG_N1, LOG_N2, WIT>;
  constexpr int N1 = C::N1, N2 = C::N2, N = C::N;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  unsigned char* base =
      reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127));
  uint64_t* bars = reinterpret_cast<uint64_t*>(base + C::OFF_BAR);
  uint64_t* a_full = bars;          // tile written (one arrival per loader warp)
  uint64_t* a_empty = bars + 1;     // pass A's MMAs done
  uint64_t* acc1_full = bars + 2;   // likewise
  uint64_t* acc1_empty = bars + 3;  // pass A's sums read (one arrival per warp of the group)
  uint64_t* b_full = bars + 4;      // pass B's operand written
  uint64_t* b_empty = bars + 5;     // pass B's MMAs done
  uint64_t* acc2_full = bars + 6;
  uint64_t* acc2_empty = bars + 7;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + 9);
  const uint32_t tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
  constexpr uint32_t kLoadWarp = kGnFold1 + kGnFold2, kMmaWarp = kLoadWarp + kGnLoad;

  if (tid == 0) {
    mbar_init(a_full, kGnLoad);
    mbar_init(a_empty, 1);
    mbar_init(acc1_full, 1);
    mbar_init(acc1_empty, kGnFold1);
    mbar_init(b_full, kGnFold1);
    mbar_init(b_empty, 1);
    mbar_init(acc2_full, 1);
    mbar_init(acc2_empty, kGnFold2);
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  for (int e = tid; e < C::TABLE / 16; e += kGnThreads) reinterpret_cast<uint4*>(base)[e] = __ldg(p.table + e);
  fence_proxy_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  auto fail = [&]() {
    record_error(p.err, LC_DEVERR_TIMEOUT);
    *abort_flag = 1;
  };
  // warp-uniform wait; false ends the role's loop
  auto wait = [&](uint64_t* bar, uint32_t parity) -> bool {
    const bool ok = mbar_wait(bar, parity);
    if (!ok) fail();
    return !__any_sync(0xffffffffu, !ok || *abort_flag);
  };
  // this CTA's k-th tile
  const uint32_t mine = p.tiles > blockIdx.x ? (p.tiles - 1 - blockIdx.x) / gridDim.x + 1 : 0;
  auto polys = [&](uint32_t tile) -> uint32_t {
    const unsigned long long left = p.count - (unsigned long long)tile * C::P;
    return left < (unsigned long long)C::P ? (uint32_t)left : (uint32_t)C::P;
  };
  int last_a = -1, last_b = -1;

  if (warp < kGnFold1) {
    // pass A: octet of columns x = (M block, x1)
    const uint32_t q = warp & 3, xl = 8 * (warp >> 2);
    const uint32_t mb = xl / N1, x0 = xl % N1;
    const uint32_t row = mb * 128 + 32 * q + lane, poly = row / N2, y2 = row % N2;
    const uint64_t* w = reinterpret_cast<const uint64_t*>(base + C::OFF_W) + x0 * N2 + y2;
    const uint32_t col = tmem + ((32 * q) << 16) + mb * 8 * N1 + x0;
    constexpr int XS = WIT ? 16 * C::P : 16;  // pass B's row: x1 P + poly or poly N1 + x1
    unsigned char* dst =
        base + C::OFF_B + (y2 >> 1) * C::LBB + (WIT ? poly * 16 : poly * N1 * 16) + x0 * XS + (y2 & 1) * 8;
    for (uint32_t k = 0; k < mine; ++k) {
      if (!wait(acc1_full, k & 1)) break;
      tc_fence_after();
      bool ok = true;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t d[8][4];
#pragma unroll
        for (int l = 0; l < 8; ++l) tmem_ld4(col + 4 * h + l * N1, d[l]);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (h == 1) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(acc1_empty);
        }
        uint64_t v[4];
        gl_fold_bytes4(d, v);
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = gl_mul_lazy(v[u], w[(4 * h + u) * N2]);
        if (h == 0 && k > 0) ok = wait(b_empty, (k - 1) & 1);  // the last tile's operand is read
        if (ok) {
#pragma unroll
          for (int u = 0; u < 4; ++u) *reinterpret_cast<uint64_t*>(dst + XS * (4 * h + u)) = v[u];
        }
      }
      if (!ok) break;
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(b_full);
    }
  } else if (warp < kLoadWarp) {
    // pass B: two octets of columns x = (M block, x2)
    const uint32_t q = warp & 3, part = (warp - kGnFold1) >> 2;
    for (uint32_t k = 0; k < mine; ++k) {
      const uint32_t tile = blockIdx.x + k * gridDim.x, np = polys(tile);
      uint32_t j0 = 0, b0 = 0;  // ring element and witness of the tile's first polynomial
      size_t place = 0;         // of this lane's polynomial in a slot
      if constexpr (WIT) {
        const unsigned long long f = (unsigned long long)tile * C::P;
        j0 = (uint32_t)(f / p.batch), b0 = (uint32_t)(f % p.batch);
        const uint32_t b = b0 + (32 * q + lane) % C::P;
        place = (size_t)(j0 + b / p.batch) * p.b_pad + b % p.batch;
      }
      if (!wait(acc2_full, k & 1)) break;
      tc_fence_after();
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        const uint32_t xl = 16 * part + 4 * h, mb = xl / N2, x0 = xl % N2;
        const uint32_t col = tmem + ((32 * q) << 16) + 256 + mb * 8 * N2 + x0;
        uint32_t d[8][4];
#pragma unroll
        for (int l = 0; l < 8; ++l) tmem_ld4(col + l * N2, d[l]);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (h == 3) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(acc2_empty);
        }
        uint64_t v[4];
        gl_fold_bytes4(d, v);
        const uint32_t row = mb * 128 + 32 * q + lane;
        if constexpr (WIT) {  // any representative: the products read bytes or reduce 160 bits
          const uint32_t poly = row % C::P, x1 = row / C::P;
          const size_t stride = (size_t)p.m * p.b_pad;
          if (poly < np) {
            uint64_t* dst = p.out + (x1 + N1 * x0) * stride + place;
#pragma unroll
            for (int u = 0; u < 4; ++u) dst[N1 * u * stride] = v[u];
          }
        } else {
          const uint32_t poly = row / N1, x1 = row % N1;
          if (poly < np) {
            uint64_t* dst = p.out + ((size_t)tile * C::P + poly) * N + x1 + N1 * x0;
#pragma unroll
            for (int u = 0; u < 4; ++u) dst[N1 * u] = gl_canon(v[u]);
          }
        }
      }
      if constexpr (WIT) {
        // the zero columns of the ring elements whose first witness is in the tile,
        // a power of two of lanes to a slot
        const uint32_t pad = p.b_pad - p.batch, t2 = tid - 32 * kGnFold1;
        if (pad) {
          const uint32_t lg = pad > 16 ? 5 : 32 - __clz(pad - 1), c0 = t2 & ((1u << lg) - 1);
          for (uint32_t j = j0 + (b0 ? 1 : 0); (unsigned long long)j * p.batch < (unsigned long long)tile * C::P + np; ++j)
            for (uint32_t t = t2 >> lg; t < (uint32_t)N; t += (32 * kGnFold2) >> lg) {
              uint64_t* z = p.out + ((size_t)t * p.m + j) * p.b_pad + p.batch;
              for (uint32_t c = c0; c < pad; c += 1u << lg) z[c] = 0;
            }
        }
      }
    }
  } else if (warp < kMmaWarp) {
    // pairs of values y1 = 2c, 2c + 1 of (poly, y2), in two halves: both loads
    // run along y2
    constexpr int PER = kGnTile / 2 / (32 * kGnLoad) / 2;  // 8 pairs per thread and half
    const uint32_t t = tid - 32 * kLoadWarp;
    for (uint32_t k = 0; k < mine; ++k) {
      const uint32_t tile = blockIdx.x + k * gridDim.x, np = polys(tile);
      uint32_t j0 = 0, b0 = 0;
      if constexpr (WIT) {
        const unsigned long long f = (unsigned long long)tile * C::P;
        j0 = (uint32_t)(f / p.batch), b0 = (uint32_t)(f % p.batch);
      }
      bool ok = true;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint64_t v[PER][2];
#pragma unroll
        for (int e = 0; e < PER; ++e) {
          const uint32_t pr = t + 32 * kGnLoad * (h * PER + e);
          const uint32_t y2 = pr % N2, c = pr / N2 % (N1 / 2), poly = pr / (N / 2);
          size_t at = (size_t)tile * C::P + poly;
          if constexpr (WIT) {
            const uint32_t b = b0 + poly;
            at = (size_t)(b % p.batch) * p.m + j0 + b / p.batch;
          }
          const uint64_t* src = p.in + at * N + 2 * c * N2 + y2;
          const bool in = poly < np;
          v[e][0] = in ? src[0] : 0;  // plain loads: out may be in
          v[e][1] = in ? src[N2] : 0;
        }
        if (h == 0 && k > 0) ok = wait(a_empty, (k - 1) & 1);
        if (ok) {
#pragma unroll
          for (int e = 0; e < PER; ++e) {
            const uint32_t pr = t + 32 * kGnLoad * (h * PER + e);
            const uint32_t y2 = pr % N2, c = pr / N2 % (N1 / 2), poly = pr / (N / 2);
            *reinterpret_cast<ulonglong2*>(base + C::OFF_A + c * C::LBA + (poly * N2 + y2) * 16) =
                make_ulonglong2(v[e][0], v[e][1]);
          }
        }
      }
      if (!ok) break;
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(a_full);
    }
  } else if (lane == 0) {
    const uint32_t va = smem_u32(base), vb = va + C::OFF_VB, ao = va + C::OFF_A, bo = va + C::OFF_B;
    auto issue_a = [&](uint32_t k) -> bool {
      if (!mbar_wait(a_full, k & 1) || (k > 0 && !mbar_wait(acc1_empty, (k - 1) & 1))) return false;
      tc_fence_after();
#pragma unroll
      for (int mb = 0; mb < 32 / N1; ++mb)
#pragma unroll
        for (int ks = 0; ks < N1 / 4; ++ks)
          mma_i8(tmem + mb * 8 * N1, umma_desc_noswz(ao + mb * 2048 + ks * 2 * C::LBA, C::LBA, 128),
                 umma_desc_noswz(va + ks * 2 * (128 * N1), 128 * N1, 128), gn_idesc(N1), ks > 0 ? 1u : 0u);
      mma_commit(acc1_full);
      mma_commit(a_empty);
      last_a = (int)k;
      return true;
    };
    auto issue_b = [&](uint32_t k) -> bool {
      if (!mbar_wait(b_full, k & 1) || (k > 0 && !mbar_wait(acc2_empty, (k - 1) & 1))) return false;
      tc_fence_after();
#pragma unroll
      for (int mb = 0; mb < 32 / N2; ++mb)
#pragma unroll
        for (int ks = 0; ks < N2 / 4; ++ks)
          mma_i8(tmem + 256 + mb * 8 * N2, umma_desc_noswz(bo + mb * 2048 + ks * 2 * C::LBB, C::LBB, 128),
                 umma_desc_noswz(vb + ks * 2 * (128 * N2), 128 * N2, 128), gn_idesc(N2), ks > 0 ? 1u : 0u);
      mma_commit(acc2_full);
      mma_commit(b_empty);
      last_b = (int)k;
      return true;
    };
    bool ok = mine == 0 || issue_a(0);
    for (uint32_t k = 0; k < mine && ok && !*abort_flag; ++k) {
      if (k + 1 < mine) ok = issue_a(k + 1);
      ok = ok && issue_b(k);
    }
    if (!ok) fail();
    // nothing may be in flight when TMEM and shared memory go
    if (last_a >= 0) mbar_wait(a_empty, (uint32_t)last_a & 1);
    if (last_b >= 0) mbar_wait(b_empty, (uint32_t)last_b & 1);
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == kMmaWarp) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
  }
}

// ------------------------------------------------------------------ tables

LC_D uint64_t gn_pow(uint64_t b, uint32_t e) {
  uint64_t r = 1;
  for (; e; e >>= 1) {
    if (e & 1) r = gl_mul(r, b);
    b = gl_mul(b, b);
  }
  return r;
}

// The table of one degree and direction, one thread per byte of VA and VB and
// per entry of W; psi of order 2n.
__global__ void __launch_bounds__(256)
    gl_ntt_table_kernel(unsigned char* table, uint64_t psi, uint64_t ninv, uint32_t log_n1, uint32_t log_n2, int inverse) {
  const uint32_t n1 = 1u << log_n1, n2 = 1u << log_n2, n = n1 * n2, order = 2 * n;
  const uint32_t sa = 64 * n1 * n1, sb = 64 * n2 * n2;
  uint32_t e = blockIdx.x * 256 + threadIdx.x;
  if (e < sa + sb) {
    const bool b = e >= sa;
    const uint32_t pts = b ? n2 : n1, at = b ? e - sa : e;
    // byte k % 16 of chunk k / 16 of row (limb, x): K index k = 8 y + lw
    const uint32_t chunk = at / (128 * pts), row = at / 16 % (8 * pts), k = 16 * chunk + at % 16;
    const uint32_t l = row / pts, x = row % pts, y = k / 8, lw = k % 8;
    uint32_t ex;  // exponent of psi, mod 2n
    if (!b) ex = inverse ? order - 2 * n2 * (x * y % n1) % order : n2 * (y * (2 * x + 1) % (2 * n1));
    else ex = inverse ? order - (2 * n1 * (x * y % n2) + n1 * x) % order : 2 * n1 * (x * y % n2);
    const uint64_t v = gl_mul(gn_pow(psi, ex % order), 1ull << (8 * lw));
    table[e] = (unsigned char)(v >> (8 * l));
    return;
  }
  e -= sa + sb;
  if (e >= n) return;
  const uint32_t x1 = e / n2, y2 = e % n2;  // stored [x1][y2]
  const uint32_t ex = inverse ? order - (2 * x1 * y2 + x1) % order : y2 * (2 * x1 + 1) % order;
  uint64_t v = gn_pow(psi, ex % order);
  if (inverse) v = gl_mul(v, ninv);
  reinterpret_cast<uint64_t*>(table + sa + sb)[e] = v;
}

static void gn_split(uint32_t log_n, uint32_t* log_n1, uint32_t* log_n2) {
  *log_n1 = (log_n + 1) / 2;
  *log_n2 = log_n / 2;
}

// per device and degree: the forward table, then the inverse one
static std::mutex g_gn_mu;
static std::atomic<unsigned char*> g_gn_table[64][11];

int gl_ntt_prepare(uint32_t log_n) {
  int dev = 0;
  if (log_n < 6 || log_n > 10) return LC_ERR_UNSUPPORTED;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
    cudaGetLastError();
    return LC_ERR_CUDA;
  }
  std::lock_guard<std::mutex> lk(g_gn_mu);
  if (g_gn_table[dev][log_n].load()) return LC_OK;
  uint32_t l1, l2;
  gn_split(log_n, &l1, &l2);
  const uint32_t bytes = (64u << (2 * l1)) + (64u << (2 * l2)) + (8u << log_n);
  unsigned char* d = nullptr;
  if (lc::dev_malloc(&d, 2 * (size_t)bytes) != cudaSuccess) {
    cudaGetLastError();
    return LC_ERR_OUT_OF_MEMORY;
  }
  const auto mul = [](uint64_t a, uint64_t b) { return (uint64_t)((unsigned __int128)a * b % kGlP); };
  uint64_t psi = 1, ninv = 1, b = 7;  // 7^((p - 1) / 2n), field.rs:195-200
  for (uint64_t e = (kGlP - 1) >> (log_n + 1); e; e >>= 1) {
    if (e & 1) psi = mul(psi, b);
    b = mul(b, b);
  }
  for (uint32_t i = 0; i < log_n; ++i) ninv = mul(ninv, (kGlP + 1) / 2);
  const uint32_t items = (64u << (2 * l1)) + (64u << (2 * l2)) + (1u << log_n);
  for (int inv = 0; inv < 2; ++inv)
    gl_ntt_table_kernel<<<(items + 255) / 256, 256>>>(d + (size_t)inv * bytes, psi, ninv, l1, l2, inv);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaStreamSynchronize(nullptr);  // any stream may use it from here on
  if (e != cudaSuccess) {
    cudaFree(d);
    return map_cuda(e);
  }
  g_gn_table[dev][log_n].store(d);
  return LC_OK;
}

template <int LOG_N1, int LOG_N2, bool WIT>
static int gn_launch(GnParams& p, const unsigned char* table, bool inverse, cudaStream_t st) {
  using C = GnCfg<LOG_N1, LOG_N2, WIT>;
  auto kern = gl_ntt_kernel<LOG_N1, LOG_N2, WIT>;
  static std::atomic<uint64_t> attr_done{0};
  const cudaError_t e = smem_attr_once(attr_done, kern, C::SMEM);
  if (e != cudaSuccess) return map_cuda(e);
  p.table = reinterpret_cast<const uint4*>(table + (inverse ? C::TABLE : 0));
  const unsigned long long tiles = (p.count + C::P - 1) / C::P;
  if (tiles >> 32) return LC_ERR_UNSUPPORTED;
  p.tiles = (uint32_t)tiles;
  kern<<<std::min<uint32_t>(p.tiles, (uint32_t)std::max(1, device_sm_count())), kGnThreads, C::SMEM, st>>>(p);
  return map_cuda(cudaGetLastError());
}

int gl_witness_ntt(uint32_t log_n, const uint64_t* w, size_t batch, uint32_t m, uint32_t b_pad, uint64_t* what_t,
                   uint32_t* err, cudaStream_t st) {
  int dev = 0;
  if ((log_n != 7 && log_n != 8) || (batch * m) << log_n < kGnMinWitness) return LC_ERR_UNSUPPORTED;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return LC_ERR_UNSUPPORTED;
  const unsigned char* table = g_gn_table[dev][log_n].load();
  if (!table) return LC_ERR_UNSUPPORTED;
  GnParams p{w, what_t, nullptr, (unsigned long long)batch * m, 0, err, m, (uint32_t)batch, b_pad};
  return log_n == 7 ? gn_launch<4, 3, true>(p, table, false, st) : gn_launch<4, 4, true>(p, table, false, st);
}

int gl_ntt(uint32_t log_n, const void* in, void* out, size_t count, bool inverse, uint32_t* err, cudaStream_t st) {
  int dev = 0;
  if (log_n < 6 || log_n > 10 || cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return LC_ERR_UNSUPPORTED;
  if (count << log_n < kGnMinValues[log_n]) return LC_ERR_UNSUPPORTED;
  const unsigned char* table = g_gn_table[dev][log_n].load();
  if (!table) return LC_ERR_UNSUPPORTED;
  GnParams p{static_cast<const uint64_t*>(in), static_cast<uint64_t*>(out), nullptr, count, 0, err, 0, 1, 0};
  switch (log_n) {
    case 6: return gn_launch<3, 3, false>(p, table, inverse, st);
    case 7: return gn_launch<4, 3, false>(p, table, inverse, st);
    case 8: return gn_launch<4, 4, false>(p, table, inverse, st);
    case 9: return gn_launch<5, 4, false>(p, table, inverse, st);
    default: return gn_launch<5, 5, false>(p, table, inverse, st);
  }
}

}  // namespace lc
