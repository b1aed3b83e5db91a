// labinius.cu -- the labinius Ajtai commitment over R_648 = Z_q[X]/Phi_1944(X).
//
// CommitmentKey::commit (lattice-labinius/src/key.rs:223-474, scalar path
// :382-474 as the specification): the witness is a stream of F162 elements;
// ring element i of chunk c lifts elements 4i..4i+3 of the chunk into the
// binary coefficients c[4m + k] = bit m of element 4i + k (binfield.rs:
// 128-143).  Per limb prime q (seven primes below 2^15, params.rs:20-30,
// :306-308) each lifted element is transformed on the limb's tree
// (scalar.rs:37-86 for q = 1 mod 1944: Phi_6 split, radix 2, 2, 3, 3, 3, 3,
// slot j = a(psi^SLOT_EXP[j]); scalar.rs:165-213 for the quadratic primes:
// Phi_6 split, radix 2, 3, 3, 3, 3 down to 324 leaves X^2 - psi'^u), then
// y += A_i (.) t (pointwise, or the per-leaf product of mul_quad_slots,
// scalar.rs:229-243).  The raw commitment yc = y mod q is decomposed into four
// R_162 slot elements (ring.rs:193-319).
//
// GPU mapping: the commitment transforms the binary elements on the INT8
// tensor cores (lb_commit_kernel, below) and a finish kernel reduces the
// column sums mod q and decomposes them; the general-input transform of the
// key derivation runs one warp per ring element on the tree itself.  Every
// transform value is reduced exactly and every product is exact, so the
// results equal the scalar reference bit for bit.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <new>
#include <vector>

#include "../../include/lattice_cuda.h"
#include "common.cuh"
#include "internal.h"
#include "tcgen05.cuh"

namespace lc {

constexpr int kLbN = 648, kLbN162 = 162, kLbQSlots = 324;
constexpr int kLbCond = 1944, kLbCondQ = 972;
constexpr int kLbTw = 326;  // twiddles of levels 1..6 of the split tree (2+4+8+24+72+216)
constexpr int kLbWarps = 8;

// Tensor-core transform of a binary ring element a = E(X^2) + X O(X^2): the
// 324 leaves j of either kind of prime need E(g_j) and O(g_j) for one node
// g_j -- a quadratic prime's leaf X^2 - g_j holds (E(g_j), O(g_j)) in slots
// 2j, 2j + 1; a splitting prime's roots come in pairs +-w_j with w_j^2 = g_j
// and values E(g_j) +- w_j O(g_j).
constexpr int kLbLeaves = kLbQSlots;
constexpr int kLbTiles = 3;            // leaf tiles, MMA M = 128 each
constexpr int kLbTileLeaves = kLbLeaves / kLbTiles;  // 108: equal tiles keep the CTAs in step
constexpr int kLbK = 352;              // K: 2 x 5 words x 32 bits, then the two elements' last 2 bits
constexpr int kLbElems = 64;           // ring elements per tile; MMA N = 128 rows (E then O)
constexpr int kLbImg = 128 * kLbK;     // one byte limb of one leaf tile; also one stage of digit rows
constexpr uint32_t kLbStoreWeight = 7;  // a tile of the kept limb counts as 7/4 of another's (share of the CTAs)
constexpr int kLbEpiWarps = 16, kLbProdWarps = 4;
constexpr int kLbTcThreads = 32 * (kLbEpiWarps + kLbProdWarps + 1);
constexpr int kLbOffB = 2 * kLbImg, kLbOffBar = kLbOffB + 2 * kLbImg;
constexpr size_t kLbSmem = 1024 + kLbOffBar + 128;
static_assert(kLbSmem <= 227 * 1024, "shared memory");
// D = s32, A = B = u8, both K-major, N = 128, M = 128
constexpr uint32_t kLbIdesc = (2u << 4) | ((128u >> 3) << 17) | ((128u >> 4) << 24);

// Per-limb constants: Shoup pairs (w, floor(w 2^32 / q)) for every twiddle.
struct LbLimb {
  uint32_t q, quad;
  uint32_t z6, z6s, om, oms;
  uint32_t tw[kLbTw], tws[kLbTw], tw2[kLbTw], tw2s[kLbTw];  // zeta, zeta^2 per (level, subring)
  uint32_t dtw[4][kLbN162];                                // decomposition factors
  uint32_t i_root, inv2;
  // per leaf of the tensor-core form: its node g_j, slots (first | second << 16) and w_j
  // with its Shoup quotient (splitting primes) or g_j (quadratic primes)
  uint32_t node[kLbLeaves], pair_slot[kLbLeaves], pair_w[kLbLeaves], pair_ws[kLbLeaves];
};

// Index maps shared by every prime (params.rs:88-97, ring.rs:68-99, params.rs:318-355).
struct LbMaps {
  uint16_t slot_648[4][kLbN162];
  uint16_t quad_class_slot[2][kLbN162];
};

__constant__ LbMaps c_lb_maps;

constexpr int kLbMaxLimbs = 7;
// one prime's tables on the device: its constants, then its transform matrices
// [tile][byte limb][128 x 352]
constexpr size_t kLbOffImg = (sizeof(LbLimb) + 255) / 256 * 256;

}  // namespace lc

struct lc_lb_key {
  size_t len_f162 = 0, nr = 0;
  uint32_t limbs = 0;
  std::vector<uint16_t> primes;
  std::vector<int16_t> a_host;  // centered rows [limbs][nr][648]
  uint32_t* d_a = nullptr;      // canonical rows by leaf [limbs][nr][324]: first slot | second << 16
  const lc::LbLimb* limb[lc::kLbMaxLimbs] = {};  // the primes' tables (device), shared by keys
  uint32_t* d_sums = nullptr;   // column sums [limbs][r][648], zero between calls
  size_t sums_bytes = 0;
  uint32_t* d_err = nullptr;    // after the rows
  uint64_t* d_in = nullptr;  // host-API staging
  size_t in_bytes = 0;
  void* d_out = nullptr;
  size_t out_bytes = 0;
};

namespace lc {

// ------------------------------------------------------------------ host tables

static uint64_t lb_pow(uint64_t b, uint64_t e, uint64_t q) {
  uint64_t r = 1;
  b %= q;
  while (e) {
    if (e & 1) r = r * b % q;
    b = b * b % q;
    e >>= 1;
  }
  return r;
}

static const int kRadix[7] = {2, 2, 2, 3, 3, 3, 3};
static const int kSub[8] = {1, 2, 4, 8, 24, 72, 216, 648};
static const int kRadixQ[6] = {2, 2, 3, 3, 3, 3};
static const int kSubQ[7] = {1, 2, 4, 12, 36, 108, 324};

// exponent of sub-ring k at a level (params.rs:73-85, :273-285)
static uint32_t sub_exp(bool quad, int level, int k) {
  if (level == 1) return quad ? (k == 0 ? 162 : 810) : (k == 0 ? 324 : 1620);
  const uint32_t p = (uint32_t)(quad ? kRadixQ[level - 1] : kRadix[level - 1]);
  const uint32_t cond = quad ? kLbCondQ : kLbCond;
  return (sub_exp(quad, level - 1, k / (int)p) + cond * ((uint32_t)k % p)) / p;
}

static bool lb_is_quad(uint32_t q) { return (q - 1) % kLbCondQ == 0 && (q - 1) % kLbCond != 0; }

static bool lb_prime_ok(uint32_t q) {
  switch (q) {
    case 2917: case 3889: case 4861: case 9721: case 12637: case 17497: case 19441: return true;
    default: return false;
  }
}

static uint32_t find_root(uint32_t q, bool quad) {  // params.rs:61-70, :262-270
  const uint64_t ord = quad ? 972 : 1944;
  for (uint64_t x = 2;; ++x)
    if (lb_pow(x, ord, q) == 1 && lb_pow(x, ord / 2, q) != 1 && lb_pow(x, ord / 3, q) != 1) return (uint32_t)x;
}

static uint32_t shoup32(uint32_t w, uint32_t q) { return (uint32_t)(((uint64_t)w << 32) / q); }

static void build_maps(LbMaps& m) {
  uint16_t slot_exp[kLbN], quad_exp[kLbQSlots], pow3[kLbN162];
  for (int j = 0; j < kLbN; ++j) slot_exp[j] = (uint16_t)sub_exp(false, 7, j);
  for (int j = 0; j < kLbQSlots; ++j) quad_exp[j] = (uint16_t)sub_exp(true, 6, j);
  int pos[486];
  std::fill(pos, pos + 486, -1);
  int n = 0;
  for (int j = 0; j < kLbN; ++j) {
    const int u = slot_exp[j], v = u % 486, t = (u - v) / 486;
    if (pos[v] < 0) {
      pos[v] = n;
      pow3[n++] = (uint16_t)v;
    }
    m.slot_648[t][pos[v]] = (uint16_t)j;
  }
  for (int s = 0; s < kLbN162; ++s)
    for (int j = 0; j < kLbQSlots; ++j) {
      if (quad_exp[j] == pow3[s]) m.quad_class_slot[0][s] = (uint16_t)j;
      if (quad_exp[j] == pow3[s] + 486) m.quad_class_slot[1][s] = (uint16_t)j;
    }
}

static void build_limb(uint32_t q, LbLimb& L) {
  const bool quad = lb_is_quad(q);
  std::memset(&L, 0, sizeof(L));
  L.q = q;
  L.quad = quad;
  const uint32_t psi = find_root(q, quad);
  L.z6 = (uint32_t)lb_pow(psi, quad ? 162 : 324, q);
  L.om = (uint32_t)lb_pow(psi, quad ? 324 : 648, q);
  L.z6s = shoup32(L.z6, q);
  L.oms = shoup32(L.om, q);
  const int levels = quad ? 5 : 6;
  int off = 0;
  for (int level = 1; level <= levels; ++level) {
    const int subs = quad ? kSubQ[level] : kSub[level];
    const int p = quad ? kRadixQ[level] : kRadix[level];
    for (int k = 0; k < subs; ++k) {
      const uint32_t z = (uint32_t)lb_pow(psi, sub_exp(quad, level, k) / (uint32_t)p, q);
      const uint32_t z2 = (uint32_t)((uint64_t)z * z % q);
      L.tw[off + k] = z;
      L.tws[off + k] = shoup32(z, q);
      L.tw2[off + k] = z2;
      L.tw2s[off + k] = shoup32(z2, q);
    }
    off += subs;
  }
  uint16_t pow3[kLbN162];
  {
    uint16_t slot_exp[kLbN];
    for (int j = 0; j < kLbN; ++j) slot_exp[j] = (uint16_t)sub_exp(false, 7, j);
    bool seen[486] = {};
    int n = 0;
    for (int j = 0; j < kLbN; ++j) {
      const int v = slot_exp[j] % 486;
      if (!seen[v]) {
        seen[v] = true;
        pow3[n++] = (uint16_t)v;
      }
    }
  }
  L.inv2 = (uint32_t)lb_pow(2, q - 2, q);
  if (quad) {
    for (int s = 0; s < kLbN162; ++s)  // inv2 * psi'^{-v}, ring.rs:248-262
      L.dtw[0][s] = (uint32_t)((uint64_t)L.inv2 * lb_pow(psi, (kLbCondQ - pow3[s]) % kLbCondQ, q) % q);
  } else {
    const uint64_t inv4 = lb_pow(4, q - 2, q);
    L.i_root = (uint32_t)lb_pow(psi, 486, q);
    for (int s = 0; s < kLbN162; ++s)  // inv4 * psi^{-v k}, ring.rs:167-187
      for (int k = 0; k < 4; ++k)
        L.dtw[k][s] = (uint32_t)(inv4 * lb_pow(psi, (kLbCond - (uint32_t)pow3[s] * k % kLbCond) % kLbCond, q) % q);
  }
}

// The leaves of the tensor-core form and their nodes g_j.
static void build_pairs(uint32_t q, LbLimb& L) {
  const bool quad = lb_is_quad(q);
  const uint32_t psi = find_root(q, quad);
  if (quad) {
    for (int j = 0; j < kLbLeaves; ++j) {
      L.node[j] = L.pair_w[j] = (uint32_t)lb_pow(psi, sub_exp(true, 6, j), q);
      L.pair_slot[j] = (uint32_t)(2 * j) | (uint32_t)(2 * j + 1) << 16;
    }
    return;
  }
  // psi^972 = -1: slots whose exponents differ by 972 hold +-w_j
  uint16_t slot_of[kLbCond] = {};
  for (int j = 0; j < kLbN; ++j) slot_of[sub_exp(false, 7, j)] = (uint16_t)j;
  int n = 0;
  for (int j = 0; j < kLbN; ++j) {
    const uint32_t e = sub_exp(false, 7, j);
    const int partner = slot_of[(e + kLbCond / 2) % kLbCond];
    if (partner < j) continue;  // seen from its partner
    const uint32_t w = (uint32_t)lb_pow(psi, e, q);
    L.node[n] = (uint32_t)((uint64_t)w * w % q);
    L.pair_slot[n] = (uint32_t)j | (uint32_t)partner << 16;
    L.pair_w[n] = w;
    L.pair_ws[n++] = shoup32(w, q);
  }
}

// c_lb_maps is constant memory of each device: uploaded once per device (one
// bit per device; devices past 63 upload on every call).
static std::mutex g_maps_mu;
static uint64_t g_maps_done = 0;

static int ensure_maps() {
  int dev = 0;
  const cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return map_cuda(e);
  const uint64_t bit = (dev >= 0 && dev < 64) ? (uint64_t)1 << dev : 0;
  std::lock_guard<std::mutex> lk(g_maps_mu);
  if (bit && (g_maps_done & bit)) return LC_OK;
  LbMaps m;
  build_maps(m);
  const int rc = map_cuda(cudaMemcpyToSymbol(c_lb_maps, &m, sizeof(m)));
  if (rc == LC_OK) g_maps_done |= bit;
  return rc;
}

// ------------------------------------------------------------------ device arithmetic

// x * w mod q, x < 2^32, w < q with ws = floor(w 2^32 / q): a representative in [0, 2q)
LC_D uint32_t lb_mulc(uint32_t x, uint32_t w, uint32_t ws, uint32_t q) { return x * w - __umulhi(x, ws) * q; }

struct LbTw {  // shared-memory copy of the limb's twiddles
  uint32_t tw[kLbTw], tws[kLbTw], tw2[kLbTw], tw2s[kLbTw];
};

// One radix-P level: NSUB sub-rings of degree DEG, twiddles at offset OFF.
// Lazy: products are representatives in [0, 2q) and differences add 2q or 4q,
// so a radix-2 level raises the bound on every value by 2q and a radix-3 level
// by 4q; the transform's values stay below 24q < 2^20.
template <int NSUB, int DEG, int P, int OFF>
LC_D void lb_level(uint32_t* v, const LbTw& T, uint32_t q, uint32_t om, uint32_t oms, uint32_t lane) {
  constexpr int M = DEG / P, BF = NSUB * M;
  const uint32_t q2 = 2 * q;
  for (int b = lane; b < BF; b += 32) {
    const int k = b / M, i = b - k * M, base = k * DEG;
    if (P == 2) {
      const uint32_t a0 = v[base + i];
      const uint32_t t = lb_mulc(v[base + M + i], T.tw[OFF + k], T.tws[OFF + k], q);
      v[base + i] = a0 + t;
      v[base + M + i] = a0 + q2 - t;
    } else {
      // a0 + w t1 + w^2 t2 = a0 - t2 + w (t1 - t2) and a0 + w^2 t1 + w t2 = a0 - t1 - w (t1 - t2)
      const uint32_t a0 = v[base + i];
      const uint32_t t1 = lb_mulc(v[base + M + i], T.tw[OFF + k], T.tws[OFF + k], q);
      const uint32_t t2 = lb_mulc(v[base + 2 * M + i], T.tw2[OFF + k], T.tw2s[OFF + k], q);
      const uint32_t u = lb_mulc(t1 + q2 - t2, om, oms, q);
      v[base + i] = a0 + t1 + t2;
      v[base + M + i] = a0 + q2 - t2 + u;
      v[base + 2 * M + i] = a0 + 2 * q2 - t1 - u;
    }
  }
  __syncwarp();
}

// The whole forward transform of one ring element in warp-private shared
// memory, canonical residues in and out.
LC_D void lb_transform(uint32_t* v, const LbTw& T, const LbLimb& L, uint32_t lane) {
  const uint32_t q = L.q;
  for (int i = lane; i < 324; i += 32) {  // Phi_6 split: (a0 + t, a0 + a1 - t), t = zeta6 a1
    const uint32_t a0 = v[i], a1 = v[i + 324];
    const uint32_t t = lb_mulc(a1, L.z6, L.z6s, q);
    v[i] = a0 + t;
    v[i + 324] = a0 + a1 + 2 * q - t;
  }
  __syncwarp();
  if (L.quad) {
    lb_level<2, 324, 2, 0>(v, T, q, L.om, L.oms, lane);
    lb_level<4, 162, 3, 2>(v, T, q, L.om, L.oms, lane);
    lb_level<12, 54, 3, 6>(v, T, q, L.om, L.oms, lane);
    lb_level<36, 18, 3, 18>(v, T, q, L.om, L.oms, lane);
    lb_level<108, 6, 3, 54>(v, T, q, L.om, L.oms, lane);
  } else {
    lb_level<2, 324, 2, 0>(v, T, q, L.om, L.oms, lane);
    lb_level<4, 162, 2, 2>(v, T, q, L.om, L.oms, lane);
    lb_level<8, 81, 3, 6>(v, T, q, L.om, L.oms, lane);
    lb_level<24, 27, 3, 14>(v, T, q, L.om, L.oms, lane);
    lb_level<72, 9, 3, 38>(v, T, q, L.om, L.oms, lane);
    lb_level<216, 3, 3, 110>(v, T, q, L.om, L.oms, lane);
  }
  // canonical: Barrett with floor(2^32 / q) leaves [0, 2q) for values < 2^20
  const uint32_t bm = 0xFFFFFFFFu / q;
  for (int x = lane; x < kLbN; x += 32) {
    uint32_t r = v[x] - __umulhi(v[x], bm) * q;
    v[x] = r >= q ? r - q : r;
  }
  __syncwarp();
}

// The two byte limbs of the matrices of the three leaf tiles, in the operand's
// shared-memory order (16-byte K chunk, row, byte).  Digit rows keep each bit
// in place: K position 32 wd + 4 s + b holds bit 8b + s of 32-bit word wd, as
// 0 or 2^s, so the matrix entry of coefficient y there is g^y 2^-s mod q.
// Element h of a parity has the words 5h .. 5h + 4 and holds the coefficients
// y = 2 m + h (m its bit); K step 10 has both elements' bits 160 and 161.
__global__ void __launch_bounds__(256) lb_image_kernel(const LbLimb* limb, uint8_t* img) {
  const uint32_t e = blockIdx.x * 256 + threadIdx.x;  // position in one byte limb's image
  const LbLimb& L = *limb;
  const uint32_t q = L.q, kpos = e / 2048 * 16 + e % 16, row = e / 16 % 128;
  const uint32_t wd = kpos / 32, s = kpos / 4 % 8, b = kpos % 4;
  const uint32_t h = wd < 10 ? wd / 5 : b, m = wd < 10 ? 32 * (wd % 5) + 8 * b + s : 160 + s;
  uint32_t v = 0;
  if (row < (uint32_t)kLbTileLeaves && h < 2 && m < (uint32_t)kLbN162) {
    uint32_t base = L.node[blockIdx.y * kLbTileLeaves + row];
    v = 1;
    for (uint32_t y = 2 * m + h; y; y >>= 1) {
      if (y & 1) v = v * base % q;  // below 2^15 each
      base = base * base % q;
    }
    for (uint32_t t = 0; t < s; ++t) v = (v & 1 ? v + q : v) / 2;
  }
  uint8_t* dst = img + (size_t)blockIdx.y * 2 * kLbImg + e;
  dst[0] = (uint8_t)v;
  dst[kLbImg] = (uint8_t)(v >> 8);
}

struct LbCommitParams {
  const uint64_t* witness;  // [r * nr][12]
  const uint32_t* a;        // [limbs][nr][324] leaf pairs
  const LbLimb* limb[kLbMaxLimbs];
  uint32_t* sums;           // [limbs][r][648]
  uint32_t* batches;        // [r * nr][648] (limb 0) or null
  uint32_t* err;
  uint32_t nr, r, total;    // total = r * nr ring elements
  uint32_t tiles;           // of 64 ring elements
  uint32_t runs0, per0;     // runs of limb 0's tiles, tiles in each
  uint32_t runs, per;       // the other limbs'
};

// x mod q in [0, 2q) for any x < 2^32, bm = floor(2^32 / q)
LC_D uint32_t lb_barrett(uint32_t x, uint32_t q, uint32_t bm) { return x - __umulhi(x, bm) * q; }
LC_D uint32_t lb_canon(uint32_t x, uint32_t q, uint32_t bm) {
  const uint32_t r = lb_barrett(x, q, bm);
  return min(r, r - q);
}
// x mod q, canonical, for any x: three 24-bit digits, 2^24 == c24 < 2^15
LC_D uint32_t lb_canon64(uint64_t x, uint32_t q, uint32_t bm, uint32_t c24) {
  const uint32_t hi = lb_canon((uint32_t)(x >> 48) * c24 + ((uint32_t)(x >> 24) & 0xFFFFFFu), q, bm);
  return lb_canon(hi * c24 + ((uint32_t)x & 0xFFFFFFu), q, bm);
}

// One epilogue warp: leaf 32 (warp & 3) + lane of the CTA's leaf tile, ring
// elements 16 (warp >> 2) .. + 16 of every tile of the run, eight at a time.
// STORE: this limb's transform is kept.
template <bool QUAD, bool STORE, class Wait, class Release>
LC_D void lb_epilogue(const LbCommitParams& p, const LbLimb& L, uint32_t k, uint32_t lt, uint32_t t0, uint32_t t1,
                      uint32_t tmem, uint32_t warp, uint32_t lane, Wait&& wait, Release&& release) {
  const uint32_t q = L.q, bm = 0xFFFFFFFFu / q, q2 = 2 * q, c24 = (1u << 24) % q;
  const uint32_t quadrant = warp & 3, grp = warp >> 2;
  const uint32_t leaf = lt * kLbTileLeaves + 32 * quadrant + lane;
  const bool mine = 32 * quadrant + lane < (uint32_t)kLbTileLeaves;
  const uint32_t slots = mine ? L.pair_slot[leaf] : 0, w = mine ? L.pair_w[leaf] : 0, ws = mine ? L.pair_ws[leaf] : 0;
  const uint32_t s0 = slots & 0xFFFFu, s1 = slots >> 16;
  const uint32_t* ak = p.a + (size_t)k * p.nr * kLbLeaves + (mine ? leaf : 0);
  const uint32_t nr = p.nr, total = p.total;
  // Sums over the column's elements.  STORE: of a0 x, a1 y (splitting) or a0 x,
  // a1 y, a0 y + a1 x (quadratic) of the canonical slots.  Otherwise nothing is
  // reduced per element: of a0 E, a1 O, a0 O, a1 E (E, O < 2^28, a < 2^15, at
  // most 2^16 elements: below 2^59), and w and q come in at the flush.
  uint64_t acc[4] = {};
  uint32_t cur = 0;      // column of the pending sums
  bool pending = false;  // warp-uniform
  auto flush = [&]() {
    uint32_t r[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) r[e] = lb_canon64(acc[e], q, bm, c24);
    uint32_t r0 = r[0], r1 = r[1];
    if (QUAD) {  // (a0 + a1 X)(x + y X) mod (X^2 - w)
      r0 = lb_canon(r[0] + w * r[1], q, bm);
      r1 = STORE ? r[2] : lb_canon(r[2] + r[3], q, bm);
    } else if (!STORE) {  // a0 (E + w O) and a1 (E - w O)
      r0 = lb_canon(r[0] + w * r[2], q, bm);
      r1 = lb_canon(r[3] + w * (q - r[1]), q, bm);
    }
    if (mine) {
      uint32_t* dst = p.sums + ((size_t)k * p.r + cur) * kLbN;
      atomicAdd(dst + s0, r0);
      atomicAdd(dst + s1, r1);
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[e] = 0;
    pending = false;
  };
  // adds elements [a, e) of the eight
  auto mac = [&](const uint32_t (&kp)[8], const uint32_t (&x)[8], const uint32_t (&y)[8], uint32_t a, uint32_t e) {
    uint32_t s0_ = 0, s1_ = 0;
    uint64_t s2_ = 0;
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const uint32_t pair = (uint32_t)u >= a && (uint32_t)u < e ? kp[u] : 0u;
      const uint32_t a0 = pair & 0xFFFFu, a1 = pair >> 16;
      if (STORE) {  // canonical: eight products stay below 8 * 19441^2 < 2^32
        s0_ += a0 * x[u];
        s1_ += a1 * y[u];
        if (QUAD) s2_ += (uint64_t)(a0 * y[u]) + a1 * x[u];
      } else {
        acc[0] += (uint64_t)a0 * x[u];
        acc[1] += (uint64_t)a1 * y[u];
        acc[2] += (uint64_t)a0 * y[u];
        acc[3] += (uint64_t)a1 * x[u];
      }
    }
    if (STORE) {
      acc[0] += s0_;
      acc[1] += s1_;
      acc[2] += s2_;
    }
  };
  // Column and element of the first of each eight, advanced by a tile at a time.
  const uint32_t step_c = kLbElems / nr, step_i = kLbElems % nr;
  uint32_t col_of[2], at[2];
  uint32_t kp[2][8];  // this tile's key pairs, loaded while the previous tile is processed
  auto load_keys = [&](int h) {
    uint32_t i = at[h];
    if (i + 8 <= nr) {
      const uint32_t* src = ak + (size_t)i * kLbLeaves;
#pragma unroll
      for (int u = 0; u < 8; ++u) kp[h][u] = __ldg(src + u * kLbLeaves);
    } else {  // rows past the last column's are loaded and not used
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        kp[h][u] = __ldg(ak + (size_t)i * kLbLeaves);
        i = i + 1 == nr ? 0 : i + 1;
      }
    }
  };
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const uint32_t f = t0 * kLbElems + 16 * grp + 8 * h;
    col_of[h] = f / nr;
    at[h] = f - col_of[h] * nr;
    load_keys(h);
  }
  for (uint32_t t = t0; t < t1; ++t) {
    const uint32_t buf = (t - t0) & 1;
    if (!wait(t - t0)) break;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint32_t f = t * kLbElems + 16 * grp + 8 * h;
      const uint32_t lim = f < total ? min(8u, total - f) : 0u;
      // E and O columns of the tile, low and high byte limb
      uint32_t x[8], y[8], xh[8], yh[8];
      const uint32_t col = tmem + ((32 * quadrant) << 16) + buf * 256 + 16 * grp + 8 * h;
      tmem_ld8(col, x);
      tmem_ld8(col + 64, y);
      tmem_ld8(col + 128, xh);
      tmem_ld8(col + 192, yh);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      if (h == 1) release(buf);
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        x[u] += xh[u] << 8;
        y[u] += yh[u] << 8;
        if (STORE) {
          x[u] = lb_barrett(x[u], q, bm);
          if (!QUAD) {  // E +- w O in (0, 4q), two conditional subtractions
            const uint32_t tw = lb_mulc(y[u], w, ws, q);
            y[u] = x[u] + q2 - tw;
            x[u] = x[u] + tw;
            x[u] = min(x[u], x[u] - q2);
            y[u] = min(y[u], y[u] - q2);
          } else {
            y[u] = lb_barrett(y[u], q, bm);
          }
          x[u] = min(x[u], x[u] - q);
          y[u] = min(y[u], y[u] - q);
        }
      }
      if (STORE && mine) {
        uint32_t* d0 = p.batches + (size_t)f * kLbN + s0;
        uint32_t* d1 = p.batches + (size_t)f * kLbN + s1;
        if (lim == 8) {
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            d0[u * kLbN] = x[u];
            d1[u * kLbN] = y[u];
          }
        } else {
#pragma unroll
          for (int u = 0; u < 8; ++u)
            if ((uint32_t)u < lim) {
              d0[u * kLbN] = x[u];
              d1[u * kLbN] = y[u];
            }
        }
      }
      // the eight elements column by column
      uint32_t c = col_of[h], i = at[h], a = 0;
      while (a < lim) {
        const uint32_t e = a + min(lim - a, nr - i);
        if (pending && c != cur) flush();
        cur = c;
        pending = true;
        if (e - a == 8)
          mac(kp[h], x, y, 0, 8);
        else
          mac(kp[h], x, y, a, e);
        a = e;
        i = 0;
        ++c;
      }
      at[h] += step_i;
      col_of[h] += step_c;
      if (at[h] >= nr) {
        at[h] -= nr;
        ++col_of[h];
      }
      if (t + 1 < t1) load_keys(h);
    }
  }
  if (pending) flush();
}

// The commitment of all columns under limb k and leaf tile blockIdx.y: a block
// takes a run of tiles of 64 ring elements of the flat sequence (column,
// element).  For every tile the two byte limbs of
//   [E; O](g_j) = sum_y g_j^y [a_2y; a_2y+1]   (u8 x u8 -> s32, K = 352)
// are exact: |D| <= 44 * 255 * 255 per byte limb (every shift s of the digit
// rows fills an eighth of K), so low + 256 high < 2^28.  Warp roles: 0-15
// reduce, store and multiply-accumulate (four per TMEM lane quadrant), 16-19
// spread the witness bits into digit rows (one thread per row), 20 loads the
// matrices, owns TMEM and issues the MMAs.  Two digit stages, two
// accumulators; all waits bounded.
//
// As butterflies in shared memory the transform was issue-bound: 427 us for
// 2^16 elements and two limbs with the base limb's transform kept.  Here a tile
// is 22 MMAs, and the epilogue is what is left: 106 us (tensor pipe 29 %, issue
// 44 %), against 27 us for the bytes of the kept transform.  A limb whose
// transform is not kept skips the reductions per element, so the kept one gets
// more of the blocks (kLbStoreWeight; equal shares took 138 us).
__global__ void __launch_bounds__(kLbTcThreads, 1) lb_commit_kernel(const __grid_constant__ LbCommitParams p) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  unsigned char* base =
      reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(base + kLbOffBar);
  uint64_t* a_full = bars;         // matrices landed
  uint64_t* b_full = bars + 1;     // [2] digit rows written (one arrival per producer warp)
  uint64_t* b_empty = bars + 3;    // [2] MMAs of the stage done
  uint64_t* acc_full = bars + 5;   // [2] accumulator complete
  uint64_t* acc_empty = bars + 7;  // [2] accumulator read (one arrival per epilogue warp)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 9);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + 10);

  const uint32_t tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
  // blocks: limb 0's runs, then the other limbs'
  const bool first = blockIdx.x < p.runs0;
  const uint32_t rest = first ? 0 : blockIdx.x - p.runs0;
  const uint32_t lt = blockIdx.y, k = first ? 0 : 1 + rest / p.runs, per = first ? p.per0 : p.per;
  const uint32_t t0 = (first ? blockIdx.x : rest % p.runs) * per, t1 = min(p.tiles, t0 + per);
  const LbLimb& L = *p.limb[k];
  if (tid == 0) {
    mbar_init(a_full, 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(&b_full[s], kLbProdWarps);
      mbar_init(&b_empty[s], 1);
      mbar_init(&acc_full[s], 1);
      mbar_init(&acc_empty[s], kLbEpiWarps);
    }
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == kLbEpiWarps + kLbProdWarps) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  auto fail = [&]() {
    record_error(p.err, LC_DEVERR_TIMEOUT);
    *abort_flag = 1;
  };
  int last_mma = -1;

  if (warp < kLbEpiWarps) {
    auto wait = [&](uint32_t it) -> bool {  // warp-uniform result: the TMEM loads are .sync.aligned
      const bool ok = mbar_wait(&acc_full[it & 1], (it >> 1) & 1);
      if (!ok) fail();
      if (__any_sync(0xffffffffu, !ok || *abort_flag)) return false;
      tc_fence_after();
      return true;
    };
    auto release = [&](uint32_t buf) {
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[buf]);
    };
    const bool store = k == 0 && p.batches;
    if (L.quad) {
      if (store) lb_epilogue<true, true>(p, L, k, lt, t0, t1, tmem, warp, lane, wait, release);
      else lb_epilogue<true, false>(p, L, k, lt, t0, t1, tmem, warp, lane, wait, release);
    } else {
      if (store) lb_epilogue<false, true>(p, L, k, lt, t0, t1, tmem, warp, lane, wait, release);
      else lb_epilogue<false, false>(p, L, k, lt, t0, t1, tmem, warp, lane, wait, release);
    }
  } else if (warp < kLbEpiWarps + kLbProdWarps) {
    // digit row: ring element row & 63 of the tile, parity row >> 6 (elements parity and parity + 2 of the four)
    const uint32_t row = tid - 32 * kLbEpiWarps, parity = row >> 6;
    for (uint32_t t = t0; t < t1; ++t) {
      const uint32_t it = t - t0, f = t * kLbElems + (row & 63);
      uint64_t wv[2][3] = {};
      if (f < p.total) {
        const uint64_t* src = p.witness + (size_t)f * 12 + 3 * parity;
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int e = 0; e < 3; ++e) wv[h][e] = __ldg(src + 6 * h + e);
      }
      bool ok = it < 2 || mbar_wait(&b_empty[it & 1], ((it >> 1) - 1) & 1);
      if (!ok) fail();
      if (__any_sync(0xffffffffu, !ok || *abort_flag)) break;
      uint4* dst = reinterpret_cast<uint4*>(base + kLbOffB + (it & 1) * kLbImg + row * 16);
#pragma unroll
      for (int wd = 0; wd < 10; ++wd) {
        const uint64_t x64 = wv[wd / 5][(wd % 5) / 2];
        const uint32_t x = (uint32_t)(((wd % 5) & 1) ? x64 >> 32 : x64);
        const uint32_t m = 0x01010101u;
        dst[(2 * wd) * 128] = make_uint4(x & m, x & (m << 1), x & (m << 2), x & (m << 3));
        dst[(2 * wd + 1) * 128] = make_uint4(x & (m << 4), x & (m << 5), x & (m << 6), x & (m << 7));
      }
      const uint32_t z = ((uint32_t)(wv[0][2] >> 32) & 3u) | ((uint32_t)(wv[1][2] >> 32) & 3u) << 8;
      dst[20 * 128] = make_uint4(z & 0x0101u, z & 0x0202u, 0u, 0u);
      dst[21 * 128] = make_uint4(0u, 0u, 0u, 0u);
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&b_full[it & 1]);
    }
  } else if (lane == 0) {
    const uint8_t* src = reinterpret_cast<const uint8_t*>(&L) + kLbOffImg + (size_t)lt * 2 * kLbImg;
    mbar_arrive_expect_tx(a_full, 2 * kLbImg);
    bulk_g2s(base, src, kLbImg, a_full);
    bulk_g2s(base + kLbImg, src + kLbImg, kLbImg, a_full);
    if (!mbar_wait(a_full, 0)) {
      fail();
      mbar_wait(a_full, 0);  // nothing may be in flight when shared memory goes
    }
    const uint32_t aa = smem_u32(base);
    for (uint32_t t = t0; t < t1 && !*abort_flag; ++t) {
      const uint32_t it = t - t0, s = it & 1;
      if (!mbar_wait(&b_full[s], (it >> 1) & 1) || (it >= 2 && !mbar_wait(&acc_empty[s], ((it >> 1) - 1) & 1))) {
        fail();
        break;
      }
      tc_fence_after();
      const uint32_t ba = smem_u32(base + kLbOffB + s * kLbImg);
#pragma unroll
      for (int l = 0; l < 2; ++l)
#pragma unroll
        for (int ks = 0; ks < kLbK / 32; ++ks)
          mma_i8(tmem + s * 256 + l * 128, umma_desc_noswz(aa + l * kLbImg + ks * 4096, 2048, 128),
                 umma_desc_noswz(ba + ks * 4096, 2048, 128), kLbIdesc, ks > 0 ? 1u : 0u);
      mma_commit(&b_empty[s]);
      mma_commit(&acc_full[s]);
      last_mma = (int)it;
    }
    if (last_mma >= 0) mbar_wait(&acc_full[last_mma & 1], (last_mma >> 1) & 1);
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == kLbEpiWarps + kLbProdWarps) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
  }
}

LC_D int16_t lb_center(uint32_t r, uint32_t q) { return r > (q - 1) / 2 ? (int16_t)((int32_t)r - (int32_t)q) : (int16_t)r; }

struct LbFinishParams {
  uint32_t* sums;     // [limbs][r][648], read and zeroed for the next call
  const LbLimb* limb[kLbMaxLimbs];
  uint32_t* raw;      // [limbs][r][648]
  int16_t* matrix;    // [4][r][limbs][162]
  uint32_t r, nlimbs;
};

__global__ void __launch_bounds__(256) lb_finish_kernel(const __grid_constant__ LbFinishParams p) {
  __shared__ uint32_t y[kLbN];
  const uint32_t c = blockIdx.x, k = blockIdx.y;
  const LbLimb& L = *p.limb[k];
  const uint32_t q = L.q;
  uint32_t* sums = p.sums + ((size_t)k * p.r + c) * kLbN;
  for (int u = threadIdx.x; u < kLbN; u += blockDim.x) {
    y[u] = sums[u] % q;
    sums[u] = 0;
    p.raw[((size_t)k * p.r + c) * kLbN + u] = y[u];
  }
  __syncthreads();
  for (int s = threadIdx.x; s < kLbN162; s += blockDim.x) {
    int16_t o[4];
    if (!L.quad) {  // length-4 inverse DFT over the class, ring.rs:193-245
      uint32_t e[4];
#pragma unroll
      for (int t = 0; t < 4; ++t) e[t] = y[c_lb_maps.slot_648[t][s]];
      const uint64_t a = e[0] + e[2], d0 = e[0] + q - e[2], cc = e[1] + e[3], d1 = e[1] + q - e[3];
      const uint64_t id = (d1 % q) * L.i_root % q;
      const uint64_t m[4] = {a + cc, d0 + q - id, a + 2ull * q - cc, d0 + id};
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) o[kk] = lb_center((uint32_t)((m[kk] % q) * L.dtw[kk][s] % q), q);
    } else {  // 2-point butterfly over the class's two leaves, ring.rs:264-306
      const int jp = c_lb_maps.quad_class_slot[0][s], jm = c_lb_maps.quad_class_slot[1][s];
#pragma unroll
      for (int kk = 0; kk < 2; ++kk) {
        const uint64_t ep = y[2 * jp + kk], em = y[2 * jm + kk];
        o[kk] = lb_center((uint32_t)((ep + em) % q * L.inv2 % q), q);
        o[kk + 2] = lb_center((uint32_t)((ep + q - em) % q * L.dtw[0][s] % q), q);
      }
    }
#pragma unroll
    for (int row = 0; row < 4; ++row) p.matrix[(((size_t)row * p.r + c) * p.nlimbs + k) * kLbN162 + s] = o[row];
  }
}

// general-input transform of `count` ring elements (key derivation, lc_lb_ntt)
__global__ void __launch_bounds__(kLbWarps * 32)
    lb_ntt_kernel(const uint32_t* __restrict__ in, uint32_t* __restrict__ out, size_t count, const LbLimb* limb) {
  __shared__ LbTw s_tw;
  __shared__ uint32_t s_v[kLbWarps][kLbN];
  const LbLimb& L = *limb;
  for (int e = threadIdx.x; e < kLbTw; e += blockDim.x) {
    s_tw.tw[e] = L.tw[e];
    s_tw.tws[e] = L.tws[e];
    s_tw.tw2[e] = L.tw2[e];
    s_tw.tw2s[e] = L.tw2s[e];
  }
  __syncthreads();
  const uint32_t warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  uint32_t* v = s_v[warp];
  for (size_t i = (size_t)blockIdx.x * kLbWarps + warp; i < count; i += (size_t)gridDim.x * kLbWarps) {
    for (int x = lane; x < kLbN; x += 32) v[x] = in[i * kLbN + x] % L.q;
    __syncwarp();
    lb_transform(v, s_tw, L, lane);
    for (int x = lane; x < kLbN; x += 32) out[i * kLbN + x] = v[x];
    __syncwarp();
  }
}

static int lb_ntt_run(const LbLimb* d_limb, const uint32_t* in, uint32_t* out, size_t count, cudaStream_t st) {
  if (count == 0) return LC_OK;
  const size_t blocks = std::min<size_t>((count + kLbWarps - 1) / kLbWarps, (size_t)std::max(1, device_sm_count()) * 8);
  lb_ntt_kernel<<<(unsigned)blocks, kLbWarps * 32, 0, st>>>(in, out, count, d_limb);
  return map_cuda(cudaGetLastError());
}

// xorshift64* of the reference (binfield.rs:158-175)
struct LbRng {
  uint64_t s;
  explicit LbRng(uint64_t seed) : s(seed * 0x9E3779B97F4A7C15ull | 1) {}
  uint64_t next() {
    uint64_t x = s;
    x ^= x >> 12;
    x ^= x << 25;
    x ^= x >> 27;
    s = x;
    return x * 0x2545F4914F6CDD1Dull;
  }
  uint32_t below(uint32_t n) { return (uint32_t)(((next() >> 32) * n) >> 32); }
};

// The tables of a prime (host) and their copy on the current device.  They depend on
// the prime alone, so they are made once (seven primes, 0.28 MB each per device) and
// kept: built for every key they made a key of 32 elements and one to three limbs
// take 0.21, 0.35 and 0.51 ms, 0.09, 0.13 and 0.18 so.
static std::mutex g_lb_mu;
static std::map<uint32_t, LbLimb> g_lb_tabs;                           // by prime
static std::map<std::pair<int, uint32_t>, const LbLimb*> g_lb_device;  // by device and prime

static int lb_prime(uint32_t q, const LbLimb** tab, const LbLimb** dev_tab) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return map_cuda(cudaGetLastError());
  std::lock_guard<std::mutex> lk(g_lb_mu);
  auto t = g_lb_tabs.find(q);
  if (t == g_lb_tabs.end()) {
    t = g_lb_tabs.emplace(q, LbLimb{}).first;
    build_limb(q, t->second);
    build_pairs(q, t->second);
  }
  *tab = &t->second;  // nodes of the map stay where they are
  const auto d = g_lb_device.find({dev, q});
  if (d != g_lb_device.end()) {
    *dev_tab = d->second;
    return LC_OK;
  }
  uint8_t* p = nullptr;
  if (lc::dev_malloc(&p, kLbOffImg + (size_t)kLbTiles * 2 * kLbImg) != cudaSuccess) {
    cudaGetLastError();
    return LC_ERR_OUT_OF_MEMORY;
  }
  cudaError_t e = cudaMemcpy(p, &t->second, sizeof(LbLimb), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    lb_image_kernel<<<dim3(kLbImg / 256, kLbTiles), 256>>>(reinterpret_cast<const LbLimb*>(p), p + kLbOffImg);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(nullptr);  // any stream may use it from here on
  if (e != cudaSuccess) {
    cudaFree(p);
    return map_cuda(e);
  }
  *dev_tab = g_lb_device[{dev, q}] = reinterpret_cast<const LbLimb*>(p);
  return LC_OK;
}

// Canonical rows on the device, one word per leaf, and the error word.
static int lb_key_finish(lc_lb_key* key, const std::vector<const LbLimb*>& tabs) {
  const size_t words = (size_t)key->limbs * key->nr * kLbLeaves;
  std::unique_ptr<uint32_t[]> canon(new (std::nothrow) uint32_t[words + 4]);
  if (!canon) return LC_ERR_OUT_OF_MEMORY;
  std::fill_n(canon.get() + words, 4, 0u);
  for (uint32_t k = 0; k < key->limbs; ++k) {
    const int32_t q = key->primes[k];
    const uint32_t* ps = tabs[k]->pair_slot;
    const auto residue = [q](int32_t x) -> uint32_t {
      x += (x >> 31) & q;
      if ((uint32_t)x >= (uint32_t)q) {  // not a centered residue
        x %= q;
        x += (x >> 31) & q;
      }
      return (uint32_t)x;
    };
    for (size_t i = 0; i < key->nr; ++i) {
      const int16_t* row = key->a_host.data() + ((size_t)k * key->nr + i) * kLbN;
      uint32_t* out = canon.get() + ((size_t)k * key->nr + i) * kLbLeaves;
      for (int j = 0; j < kLbLeaves; ++j) out[j] = residue(row[ps[j] & 0xFFFF]) | residue(row[ps[j] >> 16]) << 16;
    }
  }
  if (lc::dev_malloc(&key->d_a, (words + 4) * 4) != cudaSuccess) {
    cudaGetLastError();
    return LC_ERR_OUT_OF_MEMORY;
  }
  key->d_err = key->d_a + words;
  return map_cuda(cudaMemcpy(key->d_a, canon.get(), (words + 4) * 4, cudaMemcpyHostToDevice));
}

static int lb_key_alloc(size_t len_f162, const uint16_t* primes, uint32_t limbs, std::vector<const LbLimb*>& tabs,
                        lc_lb_key** out) {
  if (!out || !primes || limbs == 0 || limbs > (uint32_t)kLbMaxLimbs) return LC_ERR_INVALID_ARGUMENT;
  *out = nullptr;
  // key.rs:96-100: len_f162 > 0 and a multiple of 4; no limb listed twice (:102-106)
  if (len_f162 == 0 || len_f162 % 4 || len_f162 / 4 > (1u << 16)) return LC_ERR_INVALID_ARGUMENT;  // nr <= 2^16 keeps the u64 sums exact
  for (uint32_t k = 0; k < limbs; ++k) {
    if (!lb_prime_ok(primes[k])) return LC_ERR_INVALID_ARGUMENT;
    for (uint32_t j = 0; j < k; ++j)
      if (primes[j] == primes[k]) return LC_ERR_INVALID_ARGUMENT;
  }
  if (device_sm_count() <= 0) return LC_ERR_NO_DEVICE;
  int rc = ensure_maps();
  if (rc) return rc;
  lc_lb_key* key = new (std::nothrow) lc_lb_key();
  if (!key) return LC_ERR_OUT_OF_MEMORY;
  key->len_f162 = len_f162;
  key->nr = len_f162 / 4;
  key->limbs = limbs;
  key->primes.assign(primes, primes + limbs);
  tabs.resize(limbs);
  for (uint32_t k = 0; k < limbs && !rc; ++k) rc = lb_prime(primes[k], &tabs[k], &key->limb[k]);
  if (rc) {
    lc_lb_key_destroy(key);
    return rc;
  }
  *out = key;
  return LC_OK;
}

static int grow(void** p, size_t* have, size_t need) {
  if (need <= *have) return LC_OK;
  if (*p) cudaFree(*p);
  *p = nullptr;
  *have = 0;
  if (lc::dev_malloc(p, need) != cudaSuccess) {
    cudaGetLastError();
    return LC_ERR_OUT_OF_MEMORY;
  }
  *have = need;
  return LC_OK;
}

// Zeros that are there when the call returns.  On the caller's stream the memset
// would only be recorded while that stream captures, and calls outside of the graph
// would find whatever the memory held.
static int zero_now(void* p, size_t bytes) {
  cudaStream_t s = nullptr;
  cudaError_t e = cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking);
  if (e != cudaSuccess) return map_cuda(e);
  e = cudaMemsetAsync(p, 0, bytes, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  cudaStreamDestroy(s);
  return map_cuda(e);
}

}  // namespace lc

extern "C" {

LC_API int lc_lb_key_create(size_t len_f162, const uint16_t* primes, uint32_t limbs, const int16_t* a,
                            lc_lb_key** out) {
  using namespace lc;
  if (!a) return LC_ERR_INVALID_ARGUMENT;
  lc_lb_key* key = nullptr;
  std::vector<const LbLimb*> tabs;
  int rc = lb_key_alloc(len_f162, primes, limbs, tabs, &key);
  if (rc) return rc;
  key->a_host.assign(a, a + (size_t)limbs * key->nr * kLbN);
  rc = lb_key_finish(key, tabs);
  if (rc) {
    lc_lb_key_destroy(key);
    return rc;
  }
  *out = key;
  return LC_OK;
}

// CommitmentKey::random (key.rs:94-137): per limb k an xorshift64* stream
// seeded with seed ^ 0x9E3779B9 (k + 1) draws nr x 648 uniform coefficients
// below q; the rows are their transforms, centered.
LC_API int lc_lb_key_random(size_t len_f162, uint64_t seed, const uint16_t* primes, uint32_t limbs,
                            lc_lb_key** out) {
  using namespace lc;
  lc_lb_key* key = nullptr;
  std::vector<const LbLimb*> tabs;
  int rc = lb_key_alloc(len_f162, primes, limbs, tabs, &key);
  if (rc) return rc;
  const size_t per = key->nr * kLbN;
  std::vector<uint32_t> coeffs(per), t(per);
  uint32_t* d_buf = nullptr;
  if (lc::dev_malloc(&d_buf, per * 4 * 2) != cudaSuccess) {
    cudaGetLastError();
    lc_lb_key_destroy(key);
    return LC_ERR_OUT_OF_MEMORY;
  }
  key->a_host.resize((size_t)limbs * per);
  for (uint32_t k = 0; k < limbs && !rc; ++k) {
    const uint32_t q = primes[k];
    LbRng rng(seed ^ (0x9E3779B9ull * (uint64_t)(k + 1)));
    for (size_t e = 0; e < per; ++e) coeffs[e] = rng.below(q);
    rc = map_cuda(cudaMemcpy(d_buf, coeffs.data(), per * 4, cudaMemcpyHostToDevice));
    if (!rc) rc = lb_ntt_run(key->limb[k], d_buf, d_buf + per, key->nr, nullptr);
    if (!rc) rc = map_cuda(cudaMemcpy(t.data(), d_buf + per, per * 4, cudaMemcpyDeviceToHost));
    const int32_t half = (int32_t)((q - 1) / 2);
    for (size_t e = 0; e < per && !rc; ++e)
      key->a_host[(size_t)k * per + e] = (int16_t)((int32_t)t[e] > half ? (int32_t)t[e] - (int32_t)q : (int32_t)t[e]);
  }
  cudaFree(d_buf);
  if (!rc) rc = lb_key_finish(key, tabs);
  if (rc) {
    lc_lb_key_destroy(key);
    return rc;
  }
  *out = key;
  return LC_OK;
}

LC_API void lc_lb_key_destroy(lc_lb_key* key) {
  if (!key) return;
  cudaFree(key->d_a);
  cudaFree(key->d_sums);
  cudaFree(key->d_in);
  cudaFree(key->d_out);
  delete key;
}

LC_API int lc_lb_key_info(const lc_lb_key* key, size_t* len_f162, uint32_t* limbs, uint16_t* primes, int16_t* a) {
  if (!key) return LC_ERR_INVALID_ARGUMENT;
  if (len_f162) *len_f162 = key->len_f162;
  if (limbs) *limbs = key->limbs;
  if (primes) std::copy(key->primes.begin(), key->primes.end(), primes);
  if (a) std::copy(key->a_host.begin(), key->a_host.end(), a);
  return LC_OK;
}

LC_API int lc_lb_ntt(const lc_lb_key* key, uint32_t limb, const uint32_t* in, uint32_t* out, size_t count,
                     lc_stream stream) {
  using namespace lc;
  if (!key || limb >= key->limbs || ((!in || !out) && count)) return LC_ERR_INVALID_ARGUMENT;
  return lb_ntt_run(key->limb[limb], in, out, count, (cudaStream_t)stream);
}

LC_API int lc_lb_commit(lc_lb_key* key, const uint64_t* witness, uint32_t r, uint32_t* raw, int16_t* matrix,
                        uint32_t* batches, lc_stream stream) {
  using namespace lc;
  if (!key || !witness || !raw || !matrix) return LC_ERR_INVALID_ARGUMENT;
  if (r < 2 || (r & (r - 1)) || r > (1u << 15)) return LC_ERR_INVALID_ARGUMENT;  // key.rs:388-391
  const uint32_t nr = (uint32_t)key->nr;
  cudaStream_t st = (cudaStream_t)stream;
  const size_t sums = (size_t)key->limbs * r * kLbN * 4;
  if (sums > key->sums_bytes) {
    int rc = grow((void**)&key->d_sums, &key->sums_bytes, sums);
    if (!rc) rc = zero_now(key->d_sums, sums);
    if (rc) {
      key->sums_bytes = 0;  // not zero: allocated again by the next call
      return rc;
    }
  }
  static std::atomic<uint64_t> attr_done{0};
  cudaError_t e = smem_attr_once(attr_done, lb_commit_kernel, kLbSmem);
  if (e != cudaSuccess) return map_cuda(e);
  LbCommitParams p{};
  p.witness = witness;
  p.a = key->d_a;
  std::copy(key->limb, key->limb + kLbMaxLimbs, p.limb);
  p.sums = key->d_sums;
  p.batches = batches;
  p.err = key->d_err;
  p.nr = nr;
  p.r = r;
  p.total = r * nr;  // at most 2^31
  p.tiles = (p.total + kLbElems - 1) / kLbElems;
  // One CTA per SM.  A tile of limb 0 counts kLbStoreWeight / 4 tiles of another
  // limb when its transform is kept (reduced and stored per element).
  const uint32_t w0 = batches ? kLbStoreWeight : 4, sms = (uint32_t)std::max(1, device_sm_count());
  const uint32_t slots = std::max<uint32_t>(1, sms / kLbTiles), weight = w0 + 4 * (key->limbs - 1);
  const auto cut = [&](uint32_t want, uint32_t* runs, uint32_t* per) {
    *per = (p.tiles + std::max(1u, want) - 1) / std::max(1u, want);
    *runs = (p.tiles + *per - 1) / *per;
  };
  cut((slots * w0 + weight / 2) / weight, &p.runs0, &p.per0);
  cut(key->limbs > 1 ? (slots - std::min(slots, p.runs0)) / (key->limbs - 1) : 1, &p.runs, &p.per);
  lb_commit_kernel<<<dim3(p.runs0 + p.runs * (key->limbs - 1), kLbTiles), kLbTcThreads, kLbSmem, st>>>(p);
  int rc = map_cuda(cudaGetLastError());
  if (rc) return rc;
  LbFinishParams f{key->d_sums, {}, raw, matrix, r, key->limbs};
  std::copy(key->limb, key->limb + kLbMaxLimbs, f.limb);
  lb_finish_kernel<<<dim3(r, key->limbs), 256, 0, st>>>(f);
  return map_cuda(cudaGetLastError());
}

LC_API int lc_lb_key_check(lc_lb_key* key, lc_stream stream) {
  using namespace lc;
  if (!key) return LC_ERR_INVALID_ARGUMENT;
  cudaError_t e = cudaStreamSynchronize((cudaStream_t)stream);
  uint32_t flag = 0;
  if (e == cudaSuccess) e = cudaMemcpy(&flag, key->d_err, 4, cudaMemcpyDeviceToHost);
  if (e == cudaSuccess && flag) e = cudaMemset(key->d_err, 0, 4);
  if (e != cudaSuccess) return map_cuda(e);
  return flag ? LC_ERR_TIMEOUT : LC_OK;
}

// Host buffers: witness [r * len_f162][3] u64 in, raw / matrix / batches out
// (batches may be null); synchronous.
LC_API int lc_lb_commit_host(lc_lb_key* key, const uint64_t* witness, uint32_t r, uint32_t* raw, int16_t* matrix,
                             uint32_t* batches) {
  using namespace lc;
  if (!key || !witness || !raw || !matrix) return LC_ERR_INVALID_ARGUMENT;
  if (r < 2 || (r & (r - 1)) || r > (1u << 15)) return LC_ERR_INVALID_ARGUMENT;
  const size_t wbytes = (size_t)r * key->len_f162 * 24;
  const size_t raw_b = (size_t)key->limbs * r * kLbN * 4, mat_b = (size_t)4 * r * key->limbs * kLbN162 * 2;
  const size_t bat_b = batches ? (size_t)r * key->nr * kLbN * 4 : 0;
  int rc = grow((void**)&key->d_in, &key->in_bytes, wbytes);
  if (!rc) rc = grow(&key->d_out, &key->out_bytes, raw_b + mat_b + bat_b);
  if (rc) return rc;
  char* o = static_cast<char*>(key->d_out);
  rc = map_cuda(cudaMemcpy(key->d_in, witness, wbytes, cudaMemcpyHostToDevice));
  if (!rc)
    rc = lc_lb_commit(key, key->d_in, r, (uint32_t*)o, (int16_t*)(o + raw_b),
                      batches ? (uint32_t*)(o + raw_b + mat_b) : nullptr, nullptr);
  if (!rc) rc = map_cuda(cudaMemcpy(raw, o, raw_b, cudaMemcpyDeviceToHost));
  if (!rc) rc = map_cuda(cudaMemcpy(matrix, o + raw_b, mat_b, cudaMemcpyDeviceToHost));
  if (!rc && batches) rc = map_cuda(cudaMemcpy(batches, o + raw_b + mat_b, bat_b, cudaMemcpyDeviceToHost));
  return rc ? rc : lc_lb_key_check(key, nullptr);
}

// random_elems (binfield.rs:186-189): n uniform F162 elements as [n][3] u64 (host)
LC_API int lc_lb_random_elems(size_t n, uint64_t seed, uint64_t* out) {
  if (n && !out) return LC_ERR_INVALID_ARGUMENT;
  lc::LbRng rng(seed);
  for (size_t i = 0; i < n; ++i) {
    out[3 * i] = rng.next();
    out[3 * i + 1] = rng.next();
    out[3 * i + 2] = rng.next() & ((1ull << 34) - 1);
  }
  return LC_OK;
}

}  // extern "C"
