// quad50.cu -- the ~2^50 modulus class and its quadratic-slot incomplete NTT.
//
// Modulus50 / QuadSlotTables / RingConfig50 (lattice-ring/src/modulus50.rs):
// q = 2^50 - 2687 (or another two-adicity-7 prime in (2^49, 2^50)), n = 2^k
// with k in [1, 7].  X^n + 1 splits into n/2 quadratics X^2 - gamma_p; the
// forward transform is k-1 DIF levels (lo' = lo + w*hi, hi' = lo - w*hi, one
// twiddle per block), the inverse undoes each butterfly exactly
// (lo = (lo'+hi')/2, hi = (lo'-hi')/(2w)), and a ring product is the slotwise
// Karatsuba (u0 + u1 X)(v0 + v1 X) mod (X^2 - gamma) between two transforms.
//
// GPU layout: polynomials are contiguous [count][n] u64 residues.  T = n/V
// lanes own one polynomial, V = min(16, n) values each (fewer for few polynomials,
// q50_log_v_few), in registers.  Phase 0
// holds elements t + T r: the levels whose pairs are at least T apart.  The
// values change hands once, through a padded copy in the warp's shared memory,
// and phase 1 holds V consecutive elements: the remaining levels and the
// quadratic slots.  The inverse runs the same way back.
//
// Arithmetic: values are doubles that hold integers, lazily in (-8q, 8q),
// 8q < 2^53, so sums and differences are exact.  A product with a constant w,
// kept centered (|w| <= q/2) with wq = RN(w/q), is
//   h = RN(aw), l = fma(a, w, -h) (so h + l = aw exactly),
//   c = fma(a, wq, M) - M (M = 1.5 * 2^52: the integer nearest a wq),
//   r = fma(-c, q, h) + l = aw - cq exactly,
// with |r| <= q/2 + |a|/16 for |a| <= 4q (|a wq| <= 2^51).  Larger |a| take
// M = 1.5 * 2^53, which rounds to even integers: |r| <= q + |a|/16.  A forward
// butterfly (lo + r, lo - r) raises the bound on its values by |r|, and the at
// most six levels need no reduction: inputs below q reach 4.2 q after five and
// stay below 5.5 q.  In the inverse every second level, and the one before the
// last, reduces its sums: c = fma(x, 1/q, M) - M,
// fma(-c, q, x), at most q/2.  The factors 1/2 of all levels are one factor in
// the last level's constants.  Outputs become canonical as integers, so every
// output equals the reference's u64 arithmetic bit for bit.
#include <cuda_runtime.h>

#include <algorithm>
#include <new>

#include "../../include/lattice_cuda.h"
#include "common.cuh"
#include "internal.h"

namespace lc {

struct Q50Const {
  double w, wq;  // centered constant, RN(w / q)
};

// Table on the device (entries; copied into shared memory): phase-1 constants
// of the forward levels, of the inverse levels, then the leaf gammas.
constexpr int kQ50P1 = 48, kQ50Tab = 2 * kQ50P1 + 64;

// log2 of the values per lane: 16 where there are as many, and for few polynomials
constexpr int q50_log_v(int log_n) { return log_n < 4 ? log_n : 4; }
constexpr int q50_log_v_few(int log_n) { return (log_n + 1) / 2; }

}  // namespace lc

struct lc_quad50_plan {
  uint64_t q = 0, zeta = 0, generator = 0;
  uint32_t two_adicity = 0, log_n = 0;
  uint64_t gamma[64] = {};
  // phase-0 constants: level d's block i at 2^d - 1 + i; the inverse's entry 0
  // and ninv carry the factor 2^-(levels)
  lc::Q50Const fwd0[15] = {}, inv0[15] = {}, ninv = {};
  lc::Q50Const* d_tab = nullptr;  // tables of the two forms
  lc::HostPipeline staging;
};

namespace lc {

using u128 = unsigned __int128;

enum Q50Op : int { kQ50Fwd = 0, kQ50Inv_ = 1, kQ50Slot = 2, kQ50Mul = 3 };

struct Q50Params {
  const uint64_t* a;
  const uint64_t* b;
  uint64_t* out;
  size_t count;
  double q, qinv;  // qinv = RN(1/q)
  uint64_t qi;
  const Q50Const* tab;
  Q50Const fwd0[15], inv0[15], ninv;  // uniform constants, read from the parameter bank
};

constexpr double kRound52 = 6755399441055744.0;   // 1.5 * 2^52
constexpr double kRound53 = 13510798882111488.0;  // 1.5 * 2^53

LC_D double q50_load(uint64_t x) {  // exact for x < 2^52
  return __dadd_rn(__longlong_as_double((long long)(x | 0x4330000000000000ull)), -4503599627370496.0);
}

// the canonical residue of an integer in [-q, q)
LC_D uint64_t q50_store(double r, uint64_t qi) {
  const int64_t v = __double_as_longlong(__dadd_rn(r, kRound52)) - 0x4338000000000000ll;
  return (uint64_t)(v + ((v >> 63) & (int64_t)qi));
}

template <bool BIG = false>  // |a| up to 8q
LC_D double q50_mulw(double a, Q50Const w, double q) {
  constexpr double M = BIG ? kRound53 : kRound52;
  const double h = __dmul_rn(a, w.w);
  const double l = __fma_rn(a, w.w, -h);
  const double c = __dadd_rn(__fma_rn(a, w.wq, M), -M);
  return __dadd_rn(__fma_rn(-c, q, h), l);
}

// a * b for |a|, |b| <= q: |r| <= 3q/4 (the quotient of h = RN(ab) is off by at most 1/4 before rounding)
LC_D double q50_mul(double a, double b, double q, double qinv) {
  const double h = __dmul_rn(a, b);
  const double l = __fma_rn(a, b, -h);
  const double c = __dadd_rn(__fma_rn(h, qinv, kRound52), -kRound52);
  return __dadd_rn(__fma_rn(-c, q, h), l);
}

LC_D double q50_red(double x, double q, double qinv) {  // |x| < 2^53 to [-q/2, q/2]
  const double c = __dadd_rn(__fma_rn(x, qinv, kRound52), -kRound52);
  return __fma_rn(-c, q, x);
}

template <int LOG_N, int LV>
struct Q50Geo {
  static constexpr int N = 1 << LOG_N;
  static constexpr int LOG_V = LV, V = 1 << LOG_V;
  static_assert(LOG_V <= LOG_N && LOG_N <= 2 * LOG_V, "two phases");
  static constexpr int LOG_T = LOG_N - LOG_V, T = 1 << LOG_T;  // lanes per polynomial
  static constexpr int PW = 32 / T;                            // polynomials per warp
  static constexpr int WE = PW * N;                            // elements per warp (32 V)
  static constexpr int LEVELS = LOG_N - 1;
  static constexpr int LOW0 = LOG_T > 1 ? LOG_T : 1;  // phase 0: pair bits LOG_N - 1 .. LOW0
  // phase-1 constants of pair bit b: entry [j][t], j < V >> (b + 1)
  LC_HD static constexpr int p1_off(int b) {
    int off = 0;
    for (int bb = LOG_T - 1; bb > b; --bb) off += (V >> (bb + 1)) * T;
    return off;
  }
  // one pad word per 16: both sides of the exchange are free of bank conflicts
  LC_HD static constexpr int pad(int e) { return e + (e >> 4); }
  static constexpr int SLOT = WE + WE / 16 + 1;
};

// phase 0 of the forward transform: v[r] = element t + T r
template <int LOG_N, int LV>
LC_D void q50_forward0(double (&v)[Q50Geo<LOG_N, LV>::V], const Q50Params& p) {
  using Q = Q50Geo<LOG_N, LV>;
#pragma unroll
  for (int b = LOG_N - 1; b >= Q::LOW0; --b) {
    const int d = LOG_N - 1 - b, hr = 1 << (b - Q::LOG_T);
#pragma unroll
    for (int r = 0; r < Q::V; ++r) {
      if (r & hr) continue;
      const double t = q50_mulw(v[r + hr], p.fwd0[(1 << d) - 1 + (r >> (b + 1 - Q::LOG_T))], p.q);
      v[r + hr] = __dadd_rn(v[r], -t);
      v[r] = __dadd_rn(v[r], t);
    }
  }
}

// phase 1: v[r] = element V t + r
template <int LOG_N, int LV, int B>
LC_D void q50_forward1(double (&v)[Q50Geo<LOG_N, LV>::V], const Q50Const* tab, uint32_t t, double q) {
  using Q = Q50Geo<LOG_N, LV>;
  if constexpr (B >= 1) {
    constexpr int hr = 1 << B;
#pragma unroll
    for (int r = 0; r < Q::V; ++r) {
      if (r & hr) continue;
      const double x = q50_mulw<LOG_N - 1 - B == 5>(v[r + hr], tab[Q::p1_off(B) + (r >> (B + 1)) * Q::T + t], q);
      v[r + hr] = __dadd_rn(v[r], -x);
      v[r] = __dadd_rn(v[r], x);
    }
    q50_forward1<LOG_N, LV, B - 1>(v, tab, t, q);
  }
}

// Inverse butterflies of pair bit B (level number B: 1 is the first).  Inputs are
// below 2q; bounds in q of (sums, products) after the levels of n = 128: 4, 0.75;
// 0.5 (from 8), 1.5; 3, 0.7; 0.5 (from 6), 1.4; 0.5 (from 2.8), 0.7; 0.6, 0.6.
template <int LOG_N, int B>
struct Q50Inv {
  static constexpr bool kLast = B == LOG_N - 1;
  static constexpr bool kReduce = !kLast && (B % 2 == 0 || B == LOG_N - 2);
  static constexpr bool kBig = !kLast && B % 2 == 0;
};

template <int LOG_N, int B>
LC_D void q50_inv_pair(double& lo, double& hi, Q50Const w, const Q50Params& p) {
  const double s = __dadd_rn(lo, hi), d = __dadd_rn(lo, -hi);
  hi = q50_mulw<Q50Inv<LOG_N, B>::kBig>(d, w, p.q);
  if constexpr (Q50Inv<LOG_N, B>::kLast)
    lo = q50_mulw(s, p.ninv, p.q);
  else
    lo = Q50Inv<LOG_N, B>::kReduce ? q50_red(s, p.q, p.qinv) : s;
}

template <int LOG_N, int LV, int B>
LC_D void q50_inverse1(double (&v)[Q50Geo<LOG_N, LV>::V], const Q50Const* tab, uint32_t t, const Q50Params& p) {
  using Q = Q50Geo<LOG_N, LV>;
  if constexpr (B < Q::LOW0) {
#pragma unroll
    for (int r = 0; r < Q::V; ++r) {
      if (r & (1 << B)) continue;
      q50_inv_pair<LOG_N, B>(v[r], v[r + (1 << B)], tab[kQ50P1 + Q::p1_off(B) + (r >> (B + 1)) * Q::T + t], p);
    }
    q50_inverse1<LOG_N, LV, B + 1>(v, tab, t, p);
  }
}

template <int LOG_N, int LV, int B>
LC_D void q50_inverse0(double (&v)[Q50Geo<LOG_N, LV>::V], const Q50Params& p) {
  using Q = Q50Geo<LOG_N, LV>;
  if constexpr (B < LOG_N) {
    constexpr int d = LOG_N - 1 - B, hr = 1 << (B - Q::LOG_T);
#pragma unroll
    for (int r = 0; r < Q::V; ++r) {
      if (r & hr) continue;
      q50_inv_pair<LOG_N, B>(v[r], v[r + hr], p.inv0[(1 << d) - 1 + (r >> (B + 1 - Q::LOG_T))], p);
    }
    q50_inverse0<LOG_N, LV, B + 1>(v, p);
  }
}

// u <- u (*) v slotwise, (u0 + u1 X)(v0 + v1 X) mod (X^2 - gamma_p): at most 2q
template <int LOG_N, int LV>
LC_D void q50_slotwise(double (&u)[Q50Geo<LOG_N, LV>::V], double (&v)[Q50Geo<LOG_N, LV>::V], const Q50Const* tab, uint32_t t,
                       const Q50Params& p) {
  using Q = Q50Geo<LOG_N, LV>;
#pragma unroll
  for (int s = 0; s < Q::V / 2; ++s) {
    const double u0 = q50_red(u[2 * s], p.q, p.qinv), u1 = q50_red(u[2 * s + 1], p.q, p.qinv);
    const double v0 = q50_red(v[2 * s], p.q, p.qinv), v1 = q50_red(v[2 * s + 1], p.q, p.qinv);
    const double p0 = q50_mul(u0, v0, p.q, p.qinv);
    const double p1 = q50_mul(u1, v1, p.q, p.qinv);
    const double cross = q50_mul(__dadd_rn(u0, u1), __dadd_rn(v0, v1), p.q, p.qinv);
    u[2 * s] = __dadd_rn(p0, q50_mulw(p1, tab[2 * kQ50P1 + s * Q::T + t], p.q));
    u[2 * s + 1] = __dadd_rn(cross, -__dadd_rn(p0, p1));
  }
}

// Bound: FP64 issue.  A product at n = 128 is about 13 k FP64 operations (22 k
// with a conditional correction after every sum and product and two constants
// per inverse butterfly); 2^20 of them take 1.09 ms (1.97 ms before), 0.70 of the
// pipe.  16 values per lane need 128 registers, so 16 warps per SM; fetching the
// next task into registers instead of L2 spills (1.23 ms), no prefetch: 1.17 ms.
constexpr int kQ50Warps = 4, kQ50Ctas = 4;

template <int LOG_N, int LV, int OP>
__global__ void __launch_bounds__(kQ50Warps * 32, kQ50Ctas) quad50_kernel(const __grid_constant__ Q50Params p) {
  using Q = Q50Geo<LOG_N, LV>;
  constexpr int V = Q::V, T = Q::T;
  constexpr bool TWO = OP == kQ50Slot || OP == kQ50Mul;
  // which layout the operands arrive and the results leave in: 0 = t + T r, 1 = V t + r
  constexpr bool IN0 = OP == kQ50Fwd || OP == kQ50Mul, OUT0 = OP == kQ50Inv_ || OP == kQ50Mul;
  __shared__ Q50Const s_tab[kQ50Tab];
  __shared__ double s_x[kQ50Warps][Q::SLOT];
  // With fewer values per lane the tables are on their way while the first task's
  // operands are loaded; at 16 there are no registers for that (2^20 products at n =
  // 128 1107 us instead of 1070).
  constexpr bool EARLY = V < 16;
  constexpr int TAB = (kQ50Tab + kQ50Warps * 32 - 1) / (kQ50Warps * 32);
  Q50Const pre[EARLY ? TAB : 1];
  bool waiting = EARLY;
  if constexpr (EARLY) {
#pragma unroll
    for (int e = 0; e < TAB; ++e) {
      const int at = e * kQ50Warps * 32 + (int)threadIdx.x;
      pre[e] = at < kQ50Tab ? p.tab[at] : Q50Const{};
    }
  } else {
#pragma unroll
    for (int e = 0; e < TAB; ++e)
      if (e * kQ50Warps * 32 + (int)threadIdx.x < kQ50Tab)
        s_tab[e * kQ50Warps * 32 + threadIdx.x] = p.tab[e * kQ50Warps * 32 + threadIdx.x];
    __syncthreads();
  }
  auto tables = [&]() {
    waiting = false;
    if constexpr (EARLY) {
#pragma unroll
      for (int e = 0; e < TAB; ++e) {
        const int at = e * kQ50Warps * 32 + (int)threadIdx.x;
        if (at < kQ50Tab) s_tab[at] = pre[e];
      }
      __syncthreads();
    }
  };
  const uint32_t warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const uint32_t t = lane % T, poly = lane / T;
  const size_t total = p.count * Q::N;
  const size_t tasks = (p.count + Q::PW - 1) / Q::PW;
  double* x = s_x[warp];
  const uint32_t e0 = poly * Q::N + t, e1 = poly * Q::N + t * V;  // this lane's first element in either layout
  auto put = [&](const double (&v)[V], bool layout0) {
#pragma unroll
    for (int r = 0; r < V; ++r) x[Q::pad(layout0 ? e0 + T * r : e1 + r)] = v[r];
    __syncwarp();
  };
  auto get = [&](double (&v)[V], bool layout0) {
#pragma unroll
    for (int r = 0; r < V; ++r) v[r] = x[Q::pad(layout0 ? e0 + T * r : e1 + r)];
    __syncwarp();
  };
  for (size_t task = (size_t)blockIdx.x * kQ50Warps + warp; task < tasks; task += (size_t)gridDim.x * kQ50Warps) {
    const size_t base = task * Q::WE;
    const uint32_t valid = total - base < (size_t)Q::WE ? (uint32_t)(total - base) : (uint32_t)Q::WE;
    // Global accesses are coalesced: with eight lanes to a polynomial layout 0
    // is read and written in 64-byte runs as it is; the others pass through
    // the warp's copy.  Plain loads (out may alias a or b).
    auto load = [&](const uint64_t* src, double (&v)[V]) {
      if constexpr (IN0 && T == 8) {
#pragma unroll
        for (int r = 0; r < V; ++r) v[r] = e0 + T * r < valid ? q50_load(src[base + e0 + T * r]) : 0.0;
      } else {
#pragma unroll
        for (int r = 0; r < V; ++r) {
          const uint32_t e = lane + 32 * r;
          x[Q::pad(e)] = e < valid ? q50_load(src[base + e]) : 0.0;
        }
        __syncwarp();
        get(v, IN0);
      }
    };
    // the next task's operands come into L2 meanwhile (one line per lane)
    const size_t next = base + (size_t)gridDim.x * kQ50Warps * Q::WE + 16 * lane;
    if (16 * lane < Q::WE && next < total) {
      asm volatile("prefetch.global.L2 [%0];" ::"l"(p.a + next));
      if (TWO) asm volatile("prefetch.global.L2 [%0];" ::"l"(p.b + next));
    }
    double u[V], v[V];
    load(p.a, u);
    if (TWO) load(p.b, v);
    if (waiting) tables();
    if (OP == kQ50Fwd || OP == kQ50Mul) {
      q50_forward0<LOG_N, LV>(u, p);
      if (T > 1) {
        put(u, true);
        get(u, false);
      }
      q50_forward1<LOG_N, LV, Q::LOW0 - 1>(u, s_tab, t, p.q);
    }
    if (OP == kQ50Mul) {
      q50_forward0<LOG_N, LV>(v, p);
      if (T > 1) {
        put(v, true);
        get(v, false);
      }
      q50_forward1<LOG_N, LV, Q::LOW0 - 1>(v, s_tab, t, p.q);
    }
    if (TWO) q50_slotwise<LOG_N, LV>(u, v, s_tab, t, p);
    if (OP == kQ50Inv_ || OP == kQ50Mul) {
      q50_inverse1<LOG_N, LV, 1>(u, s_tab, t, p);
      if (T > 1) {
        put(u, false);
        get(u, true);
      }
      q50_inverse0<LOG_N, LV, Q::LOW0>(u, p);
    }
    if (OP == kQ50Fwd || OP == kQ50Slot || LOG_N == 1) {  // the last inverse level leaves 0.6q by itself
#pragma unroll
      for (int r = 0; r < V; ++r) u[r] = q50_red(u[r], p.q, p.qinv);
    }
    if constexpr (OUT0 && T == 8) {
#pragma unroll
      for (int r = 0; r < V; ++r)
        if (e0 + T * r < valid) p.out[base + e0 + T * r] = q50_store(u[r], p.qi);
    } else {
      put(u, OUT0);
#pragma unroll
      for (int r = 0; r < V; ++r) {
        const uint32_t e = lane + 32 * r;
        if (e < valid) p.out[base + e] = q50_store(x[Q::pad(e)], p.qi);
      }
      __syncwarp();
    }
  }
  if (waiting) tables();  // a warp without a task: the block's barrier
}

template <int LOG_N, int LV, int OP>
static int q50_launch_as(const lc_quad50_plan* plan, const uint64_t* a, const uint64_t* b, uint64_t* out, size_t count,
                         cudaStream_t st) {
  using Q = Q50Geo<LOG_N, LV>;
  const Q50Const* tab = plan->d_tab + (LV == q50_log_v(LOG_N) ? 0 : kQ50Tab);
  Q50Params p{a, b, out, count, (double)plan->q, 1.0 / (double)plan->q, plan->q, tab, {}, {}, plan->ninv};
  std::copy(plan->fwd0, plan->fwd0 + 15, p.fwd0);
  std::copy(plan->inv0, plan->inv0 + 15, p.inv0);
  const size_t tasks = (count + Q::PW - 1) / Q::PW;
  const size_t want = (tasks + kQ50Warps - 1) / kQ50Warps;
  const size_t cap = (size_t)std::max(1, device_sm_count()) * kQ50Ctas;
  quad50_kernel<LOG_N, LV, OP><<<(unsigned)std::min(want, cap), kQ50Warps * 32, 0, st>>>(p);
  return map_cuda(cudaGetLastError());
}

// Few polynomials are a matter of one lane's chain of operations: up to
// kQ50FewValues values per SM they take the fewest values per lane that two phases
// allow (n = 128 has no other split).  Products, us in a graph, 16 values per lane /
// fewer / one butterfly per lane and level through shared memory, which this kernel
// replaced: 148 of n = 16 4.76 / 2.40 / 2.75, n = 32 5.34 / 3.13 / 3.03, n = 64 5.66 /
// 2.81 / 3.27; 9472 of n = 64, past the line, 7.3 / 6.2 / 10.3.  Forward transforms:
// 148 of n = 64 3.54 / 2.24 / 2.11, and of n = 128 3.26 against 2.64.
constexpr size_t kQ50FewValues = 2048;

template <int LOG_N, int OP>
static int q50_launch(const lc_quad50_plan* plan, const uint64_t* a, const uint64_t* b, uint64_t* out,
                      size_t count, cudaStream_t st) {
  if constexpr (q50_log_v_few(LOG_N) < q50_log_v(LOG_N))
    if (count << LOG_N <= kQ50FewValues * (size_t)std::max(1, device_sm_count()))
      return q50_launch_as<LOG_N, q50_log_v_few(LOG_N), OP>(plan, a, b, out, count, st);
  return q50_launch_as<LOG_N, q50_log_v(LOG_N), OP>(plan, a, b, out, count, st);
}

template <int OP>
static int q50_dispatch(const lc_quad50_plan* plan, const uint64_t* a, const uint64_t* b, uint64_t* out,
                        size_t count, cudaStream_t st) {
  switch (plan->log_n) {
    case 1: return q50_launch<1, OP>(plan, a, b, out, count, st);
    case 2: return q50_launch<2, OP>(plan, a, b, out, count, st);
    case 3: return q50_launch<3, OP>(plan, a, b, out, count, st);
    case 4: return q50_launch<4, OP>(plan, a, b, out, count, st);
    case 5: return q50_launch<5, OP>(plan, a, b, out, count, st);
    case 6: return q50_launch<6, OP>(plan, a, b, out, count, st);
    case 7: return q50_launch<7, OP>(plan, a, b, out, count, st);
    default: return LC_ERR_INVALID_ARGUMENT;
  }
}

static int q50_run(const lc_quad50_plan* plan, int op, const uint64_t* a, const uint64_t* b, uint64_t* out,
                   size_t count, cudaStream_t st) {
  if (!plan || ((!a || !out || (op >= kQ50Slot && !b)) && count)) return LC_ERR_INVALID_ARGUMENT;
  if (count > ((size_t)1 << 36)) return LC_ERR_INVALID_ARGUMENT;
  if (count == 0) return LC_OK;
  if (device_sm_count() <= 0) return LC_ERR_NO_DEVICE;
  switch (op) {
    case kQ50Fwd: return q50_dispatch<kQ50Fwd>(plan, a, b, out, count, st);
    case kQ50Inv_: return q50_dispatch<kQ50Inv_>(plan, a, b, out, count, st);
    case kQ50Slot: return q50_dispatch<kQ50Slot>(plan, a, b, out, count, st);
    default: return q50_dispatch<kQ50Mul>(plan, a, b, out, count, st);
  }
}

// host-side exact arithmetic for the tables
static uint64_t hmul(uint64_t a, uint64_t b, uint64_t q) { return (uint64_t)((u128)a * b % q); }

static uint64_t hpow(uint64_t b, uint64_t e, uint64_t q) {
  uint64_t acc = 1 % q;
  b %= q;
  while (e) {
    if (e & 1) acc = hmul(acc, b, q);
    b = hmul(b, b, q);
    e >>= 1;
  }
  return acc;
}

static uint32_t rev_bits(uint32_t x, uint32_t bits) {
  uint32_t r = 0;
  for (uint32_t b = 0; b < bits; ++b) r |= ((x >> b) & 1u) << (bits - 1 - b);
  return r;
}

}  // namespace lc

extern "C" {

LC_API int lc_quad50_plan_create(uint64_t q, uint32_t two_adicity, uint64_t generator, uint32_t log_n,
                                 lc_quad50_plan** out) {
  using namespace lc;
  if (!out) return LC_ERR_INVALID_ARGUMENT;
  *out = nullptr;
  if (q <= ((uint64_t)1 << 49) || q >= ((uint64_t)1 << 50) || !(q & 1)) return LC_ERR_INVALID_ARGUMENT;
  if (log_n == 0 || log_n > 7) return LC_ERR_LOG_N_OUT_OF_RANGE;  // modulus50.rs:252-254
  if (two_adicity < 7) return LC_ERR_ADICITY_TOO_SMALL;           // :255-259
  const uint64_t zeta = hpow(generator, (q - 1) >> 7, q);          // root_of_unity(7), :191-197
  if (hpow(zeta, 64, q) != q - 1) return LC_ERR_GENERATOR_INVALID;  // :266-268
  lc_quad50_plan* p = new (std::nothrow) lc_quad50_plan();
  if (!p) return LC_ERR_OUT_OF_MEMORY;
  p->q = q;
  p->zeta = zeta;
  p->generator = generator;
  p->two_adicity = two_adicity;
  p->log_n = log_n;
  auto constant = [q](uint64_t w) {  // centered, below 2^49: exact
    const double c = w > q / 2 ? -(double)(q - w) : (double)w;
    return Q50Const{c, c / (double)q};
  };
  const uint64_t ninv = hpow(hpow(2, log_n - 1, q), q - 2, q);  // the levels' factors 1/2
  Q50Const tabs[2 * kQ50Tab] = {};
  p->ninv = constant(ninv);
  for (int few = 0; few < 2; ++few) {
    Q50Const* tab = tabs + few * kQ50Tab;
    const int log_v = few ? q50_log_v_few((int)log_n) : q50_log_v((int)log_n), log_t = (int)log_n - log_v;
    const int v = 1 << log_v, t = 1 << log_t;
    int p1 = 0;
    for (uint32_t d = 0; d + 1 < log_n; ++d) {  // :272-289
      const int b = (int)log_n - 1 - (int)d;    // pair bit
      for (uint32_t i = 0; i < (1u << d); ++i) {
        const uint64_t e = ((2 * (uint64_t)rev_bits(i, d) + 1) << (5 - d)) % 128;
        const uint64_t w = hpow(zeta, e, q), wi = hpow(w, q - 2, q);
        if (b >= std::max(1, log_t)) {  // the first form's entries are the second's too
          if (few) continue;
          p->fwd0[(1u << d) - 1 + i] = constant(w);
          p->inv0[(1u << d) - 1 + i] = constant(d == 0 ? hmul(wi, ninv, q) : wi);
        } else {  // block i = lane t's j-th, stored [j][t]
          const int per = v >> (b + 1), at = p1 + (int)(i % per) * t + (int)(i / per);
          tab[at] = constant(w);
          tab[kQ50P1 + at] = constant(wi);
        }
      }
      if (b < std::max(1, log_t)) p1 += (v >> (b + 1)) * t;
    }
    for (uint32_t s = 0; s < (1u << (log_n - 1)); ++s) {  // :291-296
      const uint64_t e = ((2 * (uint64_t)rev_bits(s, log_n - 1) + 1) << (7 - log_n)) % 128;
      p->gamma[s] = hpow(zeta, e, q);
      tab[2 * kQ50P1 + (int)(s % (v / 2)) * t + (int)(s / (v / 2))] = constant(p->gamma[s]);
    }
  }
  if (device_sm_count() <= 0) {
    delete p;
    return LC_ERR_NO_DEVICE;
  }
  if (lc::dev_malloc(&p->d_tab, sizeof(tabs)) != cudaSuccess) {
    cudaGetLastError();
    delete p;
    return LC_ERR_OUT_OF_MEMORY;
  }
  cudaError_t e = cudaMemcpy(p->d_tab, tabs, sizeof(tabs), cudaMemcpyHostToDevice);
  if (e != cudaSuccess) {
    cudaFree(p->d_tab);
    delete p;
    return map_cuda(e);
  }
  *out = p;
  return LC_OK;
}

LC_API void lc_quad50_plan_destroy(lc_quad50_plan* plan) {
  if (!plan) return;
  if (plan->d_tab) cudaFree(plan->d_tab);
  plan->staging.release();
  delete plan;
}

LC_API int lc_quad50_plan_info(const lc_quad50_plan* plan, uint64_t* zeta, uint64_t* slot_constants) {
  if (!plan) return LC_ERR_INVALID_ARGUMENT;
  if (zeta) *zeta = plan->zeta;
  if (slot_constants)
    for (uint32_t s = 0; s < (1u << (plan->log_n - 1)); ++s) slot_constants[s] = plan->gamma[s];
  return LC_OK;
}

LC_API int lc_quad50_forward(const lc_quad50_plan* plan, const uint64_t* in, uint64_t* out, size_t count,
                             lc_stream stream) {
  return lc::q50_run(plan, lc::kQ50Fwd, in, nullptr, out, count, (cudaStream_t)stream);
}

LC_API int lc_quad50_inverse(const lc_quad50_plan* plan, const uint64_t* in, uint64_t* out, size_t count,
                             lc_stream stream) {
  return lc::q50_run(plan, lc::kQ50Inv_, in, nullptr, out, count, (cudaStream_t)stream);
}

LC_API int lc_quad50_slotwise_mul(const lc_quad50_plan* plan, const uint64_t* a, const uint64_t* b,
                                  uint64_t* out, size_t count, lc_stream stream) {
  return lc::q50_run(plan, lc::kQ50Slot, a, b, out, count, (cudaStream_t)stream);
}

LC_API int lc_quad50_mul(const lc_quad50_plan* plan, const uint64_t* a, const uint64_t* b, uint64_t* out,
                         size_t count, lc_stream stream) {
  return lc::q50_run(plan, lc::kQ50Mul, a, b, out, count, (cudaStream_t)stream);
}

// Host buffers: chunks of about 8 MiB per operand alternate between two
// staging buffers and streams, so copies of one chunk overlap the other's kernel.
LC_API int lc_quad50_mul_host(lc_quad50_plan* plan, const uint64_t* a, const uint64_t* b, uint64_t* out,
                              size_t count) {
  using namespace lc;
  if (!plan || ((!a || !b || !out) && count)) return LC_ERR_INVALID_ARGUMENT;
  if (count == 0) return LC_OK;
  if (device_sm_count() <= 0) return LC_ERR_NO_DEVICE;
  const size_t n = (size_t)1 << plan->log_n, pb = n * 8;
  const size_t chunk = std::min(count, std::max<size_t>(1, ((size_t)8 << 20) / pb));
  HostPipeline& hp = plan->staging;
  int rc = hp.ensure(3 * chunk * pb);
  if (rc) return rc;
  size_t done = 0;
  int k = 0;
  while (done < count) {
    const size_t c = std::min(chunk, count - done);
    cudaStream_t s = hp.stream[k % HostPipeline::kSlots];
    uint64_t* da = static_cast<uint64_t*>(hp.buf[k % HostPipeline::kSlots]);
    uint64_t* db = da + chunk * n;
    uint64_t* dout = db + chunk * n;
    cudaMemcpyAsync(da, a + done * n, c * pb, cudaMemcpyHostToDevice, s);
    cudaMemcpyAsync(db, b + done * n, c * pb, cudaMemcpyHostToDevice, s);
    rc = q50_run(plan, kQ50Mul, da, db, dout, c, s);
    if (rc) break;
    cudaMemcpyAsync(out + done * n, dout, c * pb, cudaMemcpyDeviceToHost, s);
    done += c;
    ++k;
  }
  const cudaError_t e = hp.sync();
  if (rc) return rc;
  return map_cuda(e);
}

}  // extern "C"
