// sre_engine.cuh -- warp-level Walsh-Hadamard engine for the exact-SRE sweep.
//
// Mathematics (restating src/SRE.jl:424-540 and src/Helpers.jl:90 in a form that maps to
// registers).  For an X-string x the reference builds g_x(r) = Re f + Im f with
// f(r) = conj psi(r) psi(r ^ x), applies the unnormalised WHT over all n bits and sums
// F^2 and (F^2)^q.  Because f(r ^ x) = conj f(r), the n-bit transform of g splits into
// two (n-1)-bit transforms: pick a pairing bit j with x_j = 1, restrict r to the half
// V0 = {r : r_j = 0} and compress bit j away; then
//     { F(k) : k }  =  { 2 Re W(k'), 2 Im W(k') : k' }  with  W = WHT_{n-1}(f|V0)
// (Re W holds the k with even k.x, Im W the odd ones).  So one complex transform of
// 2^(n-1) points yields all 2^n values of F, with one butterfly stage and half of the
// gathers saved.  For x = 0 the pairing bit is the top bit and
//     h(r') = (|psi(r')|^2 + |psi(r'+2^(n-1))|^2,  |psi(r')|^2 - |psi(r'+2^(n-1))|^2)
// gives F = Re, Im of WHT_{n-1}(h) directly.
//
// Any GF(2)-linear relabelling of r permutes the outputs k; the sums over k do not see
// the permutation.  The two-pass kernels use this to move the pairing bit of x < 2^PB
// into the high part of the index (swap bit j with bit n-1).
//
// Data layout of one warp's tile (R complex per lane, 32R complex per warp):
//   layout A: lane l, register i  <->  element e = 32 i + l   (coalesced gathers)
//   layout B: lane l, register i  <->  element e = R l + i
// A transform over the bits held in registers needs no data movement; switching
// between A and B goes through a warp-private, XOR-swizzled shared-memory buffer
// (conflict-free 16-byte / 8-byte accesses).
#pragma once
#include "hm_common.cuh"
#ifdef HM_TMEM_EXCHANGE
#include "tmem_transpose.cuh"
#endif

namespace hm {

// ---------------------------------------------------------------------------------
// in-register butterflies over register-index bits [LO, HI)
template <int R, int LO, int HI, typename V>
__device__ __forceinline__ void reg_wht(V (&v)[R]) {
#pragma unroll
  for (int s = LO; s < HI; ++s) {
#pragma unroll
    for (int i = 0; i < R; ++i) {
      if ((i >> s) & 1) continue;
      const int k = i | (1 << s);
      const V a = v[i], b = v[k];
      v[i] = v_add(a, b);
      v[k] = v_sub(a, b);
    }
  }
}

// One butterfly of registers i and i | 1 << S.
template <int S, typename V>
__device__ __forceinline__ void bfly(V (&v)[32], int i) {
  const int k = i | (1 << S);
  const V a = v[i], b = v[k];
  v[i] = v_add(a, b);
  v[k] = v_sub(a, b);
}
// The 32-register transforms run as 4 x 8: index bits 0, 1 inside each block of four
// registers (as soon as the block has arrived), then bits 2 .. 4 inside each of the four
// classes i mod 4 (each leaves as soon as it is done), so that the loads and stores of one
// part overlap the arithmetic of another.
template <int LO, int HI, typename V>
__device__ __forceinline__ void wht_block(V (&v)[32], int b) {
#pragma unroll
  for (int i = 4 * b; i < 4 * b + 4; ++i)
    if (LO <= 0 && HI > 0 && !(i & 1)) bfly<0>(v, i);
#pragma unroll
  for (int i = 4 * b; i < 4 * b + 4; ++i)
    if (LO <= 1 && HI > 1 && !(i & 2)) bfly<1>(v, i);
}
template <int LO, int HI, typename V>
__device__ __forceinline__ void wht_class(V (&v)[32], int c) {
#pragma unroll
  for (int i = c; i < 32; i += 4)
    if (LO <= 2 && HI > 2 && !(i & 4)) bfly<2>(v, i);
#pragma unroll
  for (int i = c; i < 32; i += 4)
    if (LO <= 3 && HI > 3 && !(i & 8)) bfly<3>(v, i);
#pragma unroll
  for (int i = c; i < 32; i += 4)
    if (LO <= 4 && HI > 4 && !(i & 16)) bfly<4>(v, i);
}

// one transform bit held by lane bit `m` (a mask): every value meets its partner's
template <int R, typename V>
__device__ __forceinline__ void lane_wht(V (&v)[R], int lane, int m) {
  const float s = (lane & m) ? -1.0f : 1.0f;
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const auto px = __shfl_xor_sync(0xffffffffu, v[i].x, m);
    const auto py = __shfl_xor_sync(0xffffffffu, v[i].y, m);
    v[i].x = fma(v[i].x, (decltype(px))s, px);
    v[i].y = fma(v[i].y, (decltype(py))s, py);
  }
}

// layout A -> layout B through a warp-private buffer of 32R elements
template <int R, typename V>
__device__ __forceinline__ void transpose_ab(V (&v)[R], V *sm, int lane) {
  constexpr int LOGR = ilog2c(R);
  constexpr int SW = 128 / (int)sizeof(V) - 1;  // slots per 128-byte bank row - 1
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int e = i * 32 + lane;
    sm[e ^ ((e >> LOGR) & SW)] = v[i];
  }
  __syncwarp();
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int e = lane * R + i;
    v[i] = sm[e ^ ((e >> LOGR) & SW)];
  }
  __syncwarp();
}

// The register butterflies of layout A over bits 2 .. 4 (bits 0, 1 done by block before), the
// exchange, and those of layout B over bits LO .. 1: the classes store as they finish, the
// blocks start as they arrive.  What is left of layout B is bits 2 .. 4, by class.
template <int LO, typename V>
__device__ __forceinline__ void wht_exchange(V (&v)[32], V *sm, int lane) {
  constexpr int SW = 128 / (int)sizeof(V) - 1;
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    wht_class<2, 5>(v, c);
#pragma unroll
    for (int i = c; i < 32; i += 4) {
      const int e = i * 32 + lane;
      sm[e ^ ((e >> 5) & SW)] = v[i];
    }
  }
  __syncwarp();
#pragma unroll
  for (int b = 0; b < 8; ++b) {
#pragma unroll
    for (int i = 4 * b; i < 4 * b + 4; ++i) {
      const int e = lane * 32 + i;
      v[i] = sm[e ^ ((e >> 5) & SW)];
    }
    wht_block<LO, 2>(v, b);
  }
  __syncwarp();
}

// ---------------------------------------------------------------------------------
// Lane <-> register exchanges through tensor memory (tmem_transpose.cuh), compiled only
// with -DHM_TMEM_EXCHANGE.  A two-pass unit must move the five element bits held by the
// lane number into registers once per pass.  Through shared memory that is a 32 KB store +
// load per warp unit on the L1/shared data path, which the ring gathers and stores also
// use; through TMEM it is three (pass 1) or one to three (pass 2) store/load rounds on the
// tensor-memory path (about 3x the shared-memory rate on B200, and a separate datapath).
// Measured on B200 the exchanges give bit-identical results but make the sweep 1.5-1.7x
// slower: every round is a store, a wait, a load and a wait in series, about 700 cycles
// per warp, and 8 warps per SM cannot hide three of them per unit.  The product path
// therefore keeps the shared-memory transposes.  A CTA allocates the columns once; each
// warp uses its own 32 lanes (warp w of the CTA reaches lanes 32 (w mod 4) ..).
#ifdef HM_TMEM_EXCHANGE
template <typename T> struct TmemCols { static constexpr int value = sizeof(T) == 8 ? 128 : 64; };

__device__ __forceinline__ uint32_t tmem_cta_alloc(uint32_t *slot, int ncols) {
  if (threadIdx.x < 32) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(slot);
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s), "r"(ncols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  return *(volatile uint32_t *)slot;
}

// every warp of the CTA must have finished its TMEM accesses
__device__ __forceinline__ void tmem_cta_free(uint32_t base, int ncols) {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (threadIdx.x < 32) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(ncols) : "memory");
}

// this warp's lanes of the CTA's allocation
__device__ __forceinline__ uint32_t tmem_warp_addr(uint32_t base) {
  return base + ((uint32_t)(32 * ((threadIdx.x >> 5) & 3)) << 16);
}

// pass-1 row: lanes e0..e4 / registers e5..e9 in, registers e0..e4 out (register i =
// element bits of i), the lane number a fixed relabelling of e5..e9
__device__ __forceinline__ void tmem_row(double2 (&v)[32], uint32_t ta) { tmem_xchg_row_f64(v, ta); }
__device__ __forceinline__ void tmem_row(float2 (&v)[32], uint32_t ta) { tmem_xchg_row_f32(v, ta); }

// pass-2 tile of 2^HI rows (6 <= HI <= 10): the row bits on lanes go to registers, lowest
// row bit at register bit 0; afterwards register bits 0 .. HI - 6 hold the rows still to
// transform
template <int HI, typename V>
__device__ __forceinline__ void tmem_tile(V (&v)[32], uint32_t ta) {
  constexpr bool F64 = sizeof(V) == 16;
  if constexpr (HI == 6) {
    if constexpr (F64) tmem_xchg_tile6_f64(v, ta); else tmem_xchg_tile6_f32(v, ta);
  } else if constexpr (HI == 7) {
    if constexpr (F64) tmem_xchg_tile7_f64(v, ta); else tmem_xchg_tile7_f32(v, ta);
  } else if constexpr (HI == 8) {
    if constexpr (F64) tmem_xchg_tile8_f64(v, ta); else tmem_xchg_tile8_f32(v, ta);
  } else if constexpr (HI == 9) {
    if constexpr (F64) tmem_xchg_tile9_f64(v, ta); else tmem_xchg_tile9_f32(v, ta);
  } else if constexpr (HI == 10) {
    if constexpr (F64) tmem_xchg_tile10_f64(v, ta); else tmem_xchg_tile10_f32(v, ta);
  }
}
#endif  // HM_TMEM_EXCHANGE

// ---------------------------------------------------------------------------------
// element builders
template <typename V>
__device__ __forceinline__ V conj_mul(V a, V b) {  // conj(a) * b
  V r;
  r.x = fma(a.x, b.x, a.y * b.y);
  r.y = fma(a.x, b.y, -(a.y * b.x));
  return r;
}
template <typename V>
__device__ __forceinline__ V zero_pair(V a, V b) {  // x = 0: (|a|^2 + |b|^2, |a|^2 - |b|^2)
  const auto na = fma(a.x, a.x, a.y * a.y);
  const auto nb = fma(b.x, b.x, b.y * b.y);
  V r;
  r.x = na + nb;
  r.y = na - nb;
  return r;
}

template <typename V> __device__ __forceinline__ V ld_psi(const V *p) { return __ldg(p); }

// ---------------------------------------------------------------------------------
// moment sets: which sums a kernel accumulates besides sum F^2
enum { QS_Q2 = 1, QS_Q23 = 3, QS_GEN = 0 };
template <int QS> struct QSet {
  static constexpr int NQ = (QS == QS_Q2) ? 1 : (QS == QS_Q23 ? 2 : 4);
};

struct QParams {
  double q[4];
  double scale[4];  // 4^q
  int nq;
  int direct;  // one q, an integer or a half-integer (half_integer_q)
};

// (F^2)^q with 2q an integer is |F| to an integer power.  q = 8.5 is left to pow(): its four
// squarings in a row, each doubling the error before it, end above pow's (rms 4.4e-16 of a value
// against 4.0e-16; 0.77 to 1.0 times the errors of squaring F^2 and of pow at all other q).
__host__ __device__ inline bool half_integer_q(double q) {
  return 2.0 * q == floor(2.0 * q) && q >= 1.0 && q <= 16.0 && q != 8.5;
}

inline void set_qparams(QParams &qp, const double *q, int nq) {
  qp.nq = nq;
  qp.direct = nq == 1 && half_integer_q(q[0]);
  for (int i = 0; i < 4; ++i) {
    qp.q[i] = i < nq ? q[i] : 2.0;
    qp.scale[i] = pow(4.0, qp.q[i]);
  }
}

// r = f^2 -> |f|^(2q), half_integer_q(q), N values side by side: the bits of the exponent 2q
// from the second one down, square and multiply by f, which has no rounding of its own.
template <int N>
__device__ __forceinline__ void pow_half(const double (&f)[N], double (&r)[N], double q) {
  const int e = (int)(2.0 * q);
  int b = 30 - __clz(e);
#pragma unroll 1
  while (true) {
    if ((e >> b) & 1) {
#pragma unroll
      for (int t = 0; t < N; ++t) r[t] *= f[t];
    }
    if (--b < 0) break;
#pragma unroll
    for (int t = 0; t < N; ++t) r[t] *= r[t];
  }
  if (e & 1) {
#pragma unroll
    for (int t = 0; t < N; ++t) r[t] = fabs(r[t]);
  }
}

template <int N> __device__ __forceinline__ double tree_sum(const double (&v)[N]) {
  double s[N];
#pragma unroll
  for (int t = 0; t < N; ++t) s[t] = v[t];
#pragma unroll
  for (int w = N / 2; w > 0; w >>= 1)
#pragma unroll
    for (int t = 0; t < w; ++t) s[t] += s[t + w];
  return s[0];
}

// Generic Renyi indices, per-lane sums of F^2 and (F^2)^q of the R complex registers.
//   one half-integer q (qp.direct): from the registers, 16 values at a time (FP32: 8, for
//     its 128 registers), so that the powers are independent chains over the FP64 latency; the
//     exponent is uniform over the grid.  A step of the loop over its bits is one product per
//     value.  FP64 on B200, all 2^n X-strings: n = 13 q = 4 318 -> 149 us (staged, four chains),
//     q = 2.5 1.50 ms -> 151 us (pow); n = 11 q = 4 52 -> 27 us; n = 20 q = 4 7.2 -> 4.5 us each.
//     FP32, us per X-string, staged -> this: n = 13 q = 4 0.053 -> 0.014, n = 18 1.53 -> 0.58, n = 20
//     7.2 -> 2.6, n = 22 45 -> 29, n = 24 162 -> 134.  F^2 is summed before it is raised, in place.
//     Error of the sums against extended precision, n = 6 .. 11: 7e-16 at q = 2.5 (pow 13e-16).
//     (A list of several q would keep all values and the sums in registers, which spill.)
template <int R, typename V>
__device__ __forceinline__ void lane_moments_direct(const V (&v)[R], double *s, const QParams &qp) {
  constexpr int N = sizeof(V) == 16 ? 16 : 8;
  double a2 = 0.0, ag = 0.0;
#pragma unroll
  for (int c = 0; c < 2 * R / N; ++c) {
    double f[N], r[N];
#pragma unroll
    for (int t = 0; t < N; ++t) {
      f[t] = (double)(t & 1 ? v[(c * N + t) / 2].y : v[(c * N + t) / 2].x);
      r[t] = f[t] * f[t];
    }
    a2 += tree_sum(r);
    pow_half(f, r, qp.q[0]);
    ag += tree_sum(r);
  }
  s[0] = a2;
  s[1] = ag;
#pragma unroll
  for (int t = 1; t < 4; ++t) s[1 + t] = 0.0;
}

//   others: the F values go through the warp's own shared buffer (sm[lane + 32 t], NV of
//     them), so that the pow() evaluations run in a rolled loop, four chains at a time.
template <int NV, typename T>
__device__ __noinline__ void lane_moments_gen(const T *sm, int lane, double *s, const QParams &qp) {
  double a2 = 0.0, ag[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 1
  for (int t0 = 0; t0 < NV; t0 += 4) {
    double f[4], y[4], r[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      f[t] = (double)sm[lane + 32 * (t0 + t)];
      y[t] = f[t] * f[t];
    }
    a2 += (y[0] + y[1]) + (y[2] + y[3]);
#pragma unroll 1
    for (int k = 0; k < qp.nq; ++k) {
      const double q = qp.q[k];
      if (half_integer_q(q)) {
#pragma unroll
        for (int t = 0; t < 4; ++t) r[t] = y[t];
        pow_half(f, r, q);
      } else {
#pragma unroll
        for (int t = 0; t < 4; ++t) r[t] = pow(y[t], q);
      }
      ag[k] += (r[0] + r[1]) + (r[2] + r[3]);
    }
  }
  s[0] = a2;
#pragma unroll
  for (int t = 0; t < 4; ++t) s[1 + t] = ag[t];
}

// Per-lane sums of F^2 and of (F^2)^q over the R complex registers (2R values of F/2
// for x != 0; the caller applies the 4 / 4^q scale), plain FP64 sums in a fixed order.
// Both precisions take the powers and the sums in FP64: an FP32 value of F converts to
// double exactly, so the FP32 path's only roundings are those of f and of the butterflies.
// NA interleaved accumulators per sum (value j goes to accumulator j mod NA, combined
// pairwise at the end) keep the dependent-add chains short; the order is fixed.
template <int R, int QS, typename V>
__device__ __forceinline__ void lane_moments(const V (&v)[R], double *s, const QParams &qp, V *sm, int lane) {
  if constexpr (QS == QS_GEN) {
    if (qp.direct) {
      lane_moments_direct(v, s, qp);
      return;
    }
    auto *f = &sm->x;
#pragma unroll
    for (int i = 0; i < R; ++i) {
      f[lane + 32 * (2 * i)] = v[i].x;
      f[lane + 32 * (2 * i + 1)] = v[i].y;
    }
    lane_moments_gen<2 * R>(f, lane, s, qp);
    __syncwarp();
    return;
  } else {
    constexpr int NA = 4;
    double a2[NA], a4[NA], a6[NA];
#pragma unroll
    for (int t = 0; t < NA; ++t) a2[t] = a4[t] = a6[t] = 0.0;
#pragma unroll
    for (int i = 0; i < R; ++i) {
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const double f = c ? (double)v[i].y : (double)v[i].x;
        const double y = f * f;
        const int t = (2 * i + c) % NA;
        a2[t] += y;
        a4[t] = fma(y, y, a4[t]);
        if constexpr (QS == QS_Q23) a6[t] = fma(y * y, y, a6[t]);
      }
    }
#pragma unroll
    for (int w = NA / 2; w > 0; w >>= 1)
#pragma unroll
      for (int t = 0; t < w; ++t) {
        a2[t] += a2[t + w];
        a4[t] += a4[t + w];
        a6[t] += a6[t + w];
      }
    s[0] = a2[0];
    s[1] = a4[0];
    if constexpr (QS == QS_Q23) s[2] = a6[0];
  }
}

// Sums of one quad of values before its last two butterfly levels.  With c_d = sum_e u_e
// u_(e^d) the four outputs satisfy sum F^2 = 4 c_0 and sum F^4 = 4 (c_0^2 + c_1^2 + c_2^2 +
// c_3^2) (F_k^2 = sum_d (-1)^(k.d) c_d, Parseval over k): 15 operations for the four values
// instead of 8 for the two levels and 12 for the powers.
struct QuadSums {
  double a2[2] = {0.0, 0.0}, m0[2] = {0.0, 0.0}, h1 = 0.0, h2 = 0.0, h3 = 0.0;
  __device__ __forceinline__ void add(int t, double u0, double u1, double u2, double u3) {
    const double c0 = fma(u0, u0, fma(u1, u1, fma(u2, u2, u3 * u3)));
    const double c1 = fma(u0, u1, u2 * u3), c2 = fma(u0, u2, u1 * u3), c3 = fma(u0, u3, u1 * u2);
    a2[t] += c0;
    m0[t] = fma(c0, c0, m0[t]);
    h1 = fma(c1, c1, h1);
    h2 = fma(c2, c2, h2);
    h3 = fma(c3, c3, h3);
  }
  __device__ __forceinline__ void get(double *s) const {
    s[0] = 4.0 * (a2[0] + a2[1]);
    s[1] = 4.0 * ((m0[0] + m0[1]) + 4.0 * ((h1 + h2) + h3));
  }
};

// The same with sum F^6: sum_k (sum_d (-1)^(k.d) c_d)^3 keeps the triples with d1 ^ d2 ^ d3 = 0,
// 4 (c_0^3 + 3 c_0 (c_1^2 + c_2^2 + c_3^2) + 6 c_1 c_2 c_3).  Here c1 .. c3 are halves of c_1 ..
// c_3.  21 operations for the four values instead of 8 for the two levels and 20 for the powers.
// FP64 on B200, q = 2 and 3: n = 13 143 -> 136 us, n = 14 594 -> 547, n = 20 4.00 -> 3.85 each.
// Error of the q = 3 sum against extended precision, n = 11, 12: 6e-16 (powers: 9e-16).
struct CubeSums {
  double a2[2] = {0.0, 0.0}, m4[2] = {0.0, 0.0}, m6[2] = {0.0, 0.0}, m111[2] = {0.0, 0.0};
  __device__ __forceinline__ void add(int t, double u0, double u1, double u2, double u3) {
    const double c0 = fma(u0, u0, fma(u1, u1, fma(u2, u2, u3 * u3)));
    const double c1 = fma(u0, u1, u2 * u3), c2 = fma(u0, u2, u1 * u3), c3 = fma(u0, u3, u1 * u2);
    const double h = fma(c1, c1, fma(c2, c2, c3 * c3)), w = c0 * c0;
    a2[t] += c0;
    m4[t] += fma(4.0, h, w);
    m6[t] = fma(c0, fma(12.0, h, w), m6[t]);
    m111[t] = fma(c1 * c2, c3, m111[t]);
  }
  __device__ __forceinline__ void get(double *s) const {
    s[0] = 4.0 * (a2[0] + a2[1]);
    s[1] = 4.0 * (m4[0] + m4[1]);
    s[2] = 4.0 * ((m6[0] + m6[1]) + 48.0 * (m111[0] + m111[1]));
  }
};
template <int QS> struct LevelSums;
template <> struct LevelSums<QS_Q2> : QuadSums {};
template <> struct LevelSums<QS_Q23> : CubeSums {};

// sums of 32 complex registers whose register bits LO .. 4 are still to transform (bits below
// 2 done): bit 2 if it is one of them, then quads over bits 3 and 4
template <int QS, int LO, typename V>
__device__ __forceinline__ void quad_moments(V (&v)[32], double *s) {
  LevelSums<QS> q;
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    if constexpr (LO <= 2) wht_class<2, 3>(v, c);
#pragma unroll
    for (int i = c; i < 8; i += 4) {
      q.add(0, v[i].x, v[i + 8].x, v[i + 16].x, v[i + 24].x);
      q.add(1, v[i].y, v[i + 8].y, v[i + 16].y, v[i + 24].y);
    }
  }
  q.get(s);
}

// scale of sum (F^2)^q for one X-string: F = 2 W (x != 0) or W (x = 0)
template <int QS>
__device__ __forceinline__ double q_scale(int t, bool xzero, const QParams &qp) {
  if (xzero) return 1.0;
  if constexpr (QS == QS_Q2) return 16.0;
  if constexpr (QS == QS_Q23) return t == 0 ? 16.0 : 64.0;
  return qp.scale[t];
}

// ---------------------------------------------------------------------------------
// X-string bookkeeping for the two-pass engine.  Pass 1 pairs rows of the high index
// part, so the pairing bit jt of x must be >= PB.  For 1 <= x < 2^PB the kernel reads a
// copy of psi with bits j (the highest set bit of x) and n-1 swapped, on which the
// relabelled string xt = x ^ 2^j ^ 2^(n-1) has its pairing bit at n-1.  x = 0 is not
// handled by the two-pass kernel (its F is the plain transform of |psi|^2).
struct XInfo {
  uint64_t xt;  // effective x after the relabelling (pairing bit in the high part)
  int jt;       // pairing bit of xt
  int sw;       // relabelling: read the copy with bits sw and n-1 swapped (or -1)
  int active;   // Gray index inside the requested range and x != 0
  int zero = 0;  // x = 0 inside the range, built with the top-bit pairing (set by the caller)
};

__device__ __forceinline__ XInfo make_xinfo(uint64_t k, uint64_t k_end, int n, int pb) {
  XInfo xi;
  const uint64_t x = gray_code(k);
  xi.active = (k < k_end) && (x != 0);
  xi.zero = 0;
  xi.sw = -1;
  xi.xt = x;
  xi.jt = x ? 63 - __clzll((long long)x) : n - 1;
  if (x != 0 && xi.jt < pb) {
    xi.sw = xi.jt;
    xi.xt = (x ^ (1ull << xi.jt)) | (1ull << (n - 1));
    xi.jt = n - 1;
  }
  return xi;
}

// Pass 1: gather + build row rho of the (n-1)-bit index of x; its low PB bits are transformed
// next (p1_unit, p1_unit_tma).
template <int R, typename V>
__device__ __forceinline__ void p1_build(V (&v)[R], const V *__restrict__ psi, const XInfo &xi, uint64_t rho, int lane) {
  constexpr int PB = ilog2c(R) + 5;
  if (xi.zero) {
    // x = 0: f(r) = |psi(r)|^2 paired on the top bit (jt = n - 1),
    // h = (|a|^2 + |b|^2, |a|^2 - |b|^2) with a = psi(r), b = psi(r + 2^(n-1))
    const V *rowA = psi + (rho << PB);
    const V *rowB = rowA + (1ull << xi.jt);
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const uint32_t e = (uint32_t)(i * 32 + lane);
      v[i] = zero_pair(ld_psi(rowA + e), ld_psi(rowB + e));
    }
    return;
  }
  const uint64_t rH = insert0(rho, xi.jt - PB);
  const uint64_t sH = rH ^ (xi.xt >> PB);
  const uint32_t xL = (uint32_t)(xi.xt & ((1ull << PB) - 1ull));
  const V *rowA = psi + (rH << PB);
  const V *rowB = psi + (sH << PB);
  // both rows straight into registers (the partner permuted by the low bits of x)
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const uint32_t e = (uint32_t)(i * 32 + lane);
    v[i] = conj_mul(ld_psi(rowA + e), ld_psi(rowB + (e ^ xL)));
  }
}

// Ring layout of one X-string's intermediate (2^(n-1) complex): tile-major,
//   inter_x[t * 2^(HI+LOGC) + row * C + c]  for pass-2 tile t, row, column c < C,
// so that a pass-2 tile is one contiguous 2^PB-element block and pass 1 writes whole
// 32-byte sectors (C >= 2).
// Hook run by every lane right before a pass-1 unit's first global store (the stage
// kernels wait there for the previous stage); the default does nothing.
struct NoHook {
  __device__ __forceinline__ void operator()() const {}
};

template <int R, int HI, typename V, typename Pre = NoHook>
__device__ __forceinline__ void p1_unit(const V *__restrict__ psi, const XInfo &xi, uint64_t rho,
                                        V *__restrict__ inter_x, V *sm, int lane, const Pre &pre = Pre()) {
  constexpr int LOGR = ilog2c(R), PB = LOGR + 5, LOGC = PB - HI;
  V v[R];
  p1_build(v, psi, xi, rho, lane);
  reg_wht<R, 0, LOGR>(v);  // element bits 5 .. PB-1
  transpose_ab<R>(v, sm, lane);
  reg_wht<R, 0, 5>(v);  // element bits 0 .. 4
  pre();
  // register i of lane l holds element k = R l + i; it is stored at position p = 32 i + l
  // of the row (any fixed relabelling of k is invisible to the moment sums)
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const uint32_t p = (uint32_t)(i * 32 + lane);
    const uint32_t t = p >> LOGC, c = p & ((1u << LOGC) - 1u);
    __stcg(inter_x + (((size_t)t << (HI + LOGC)) + (rho << LOGC) + c), v[i]);
  }
}

// ---------------------------------------------------------------------------------
// Pass-1 output through the tensor-memory-access unit.  The row's 2^PB positions land in
// 2^PB / C different pass-2 tiles, C positions each (C = 2 at n = 20): a warp-wide
// st.global of them touches 16 cache lines per instruction.  Instead the warp writes the
// row to its shared buffer in position order (conflict-free) and one thread issues
// tensor stores that scatter it to the tile-major ring (no multicast; the ring is this
// GPU's memory).  The 4-D tensor view of the ring, in scalars: d0 = the 2C scalars of a
// tile row, d1 = the 2^HI rows, d2 = the 2^PB / C tiles, d3 = the 2X (slot, X-string)
// pairs; boxes are {b0, 1, b2, 1}.
struct TmaGeom {
  int box0;  // scalars per box along d0 (2C, or 256 when 2C > 256)
  int nb0;   // boxes along d0 per tile (2C / box0)
  int box2;  // tiles per box (1 when nb0 > 1)
  int nb2;   // box groups along the tiles
  int C;     // positions per tile row
};

__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void tma_store_4d(const void *tmap, const void *smem_src, int c0, int c1, int c2, int c3) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem_src);
  asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5}], [%1];" ::"l"(tmap),
               "r"(s), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
               : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// the shared-memory source of every committed store has been read
__device__ __forceinline__ void bulk_wait_read_all() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
// every committed store has completed
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

// As p1_unit, with the row leaving through the warp's shared buffer and tensor stores.
// The caller waits for the stores to have read the buffer (bulk_wait_read_all on lane 0,
// then __syncwarp) before the buffer's next use.
template <int R, int HI, bool TM, typename V, typename Pre = NoHook, typename Ready = NoHook>
__device__ __forceinline__ void p1_unit_tma(const V *__restrict__ psi, const XInfo &xi, uint64_t rho, V *sm, int lane,
                                            const void *tmap, const TmaGeom &g, int xcoord, uint32_t ta,
                                            const Pre &pre = Pre(), const Ready &ready = Ready()) {
  constexpr int LOGR = ilog2c(R);
  V v[R];
  p1_build(v, psi, xi, rho, lane);  // registers only (no shared memory)
#ifdef HM_TMEM_EXCHANGE
  reg_wht<R, 0, LOGR>(v);
  ready();  // the shared buffer is free from here on
  static_assert(TM && R == 32, "the TMEM exchanges are generated for 32 values per lane");
  tmem_row(v, ta);
  reg_wht<R, 0, 5>(v);
#pragma unroll
  for (int i = 0; i < R; ++i) sm[i * 32 + lane] = v[i];
#else
  (void)ta;
  static_assert(R == 32 && LOGR == 5, "32 values per lane");
#pragma unroll
  for (int b = 0; b < 8; ++b) wht_block<0, 2>(v, b);
  ready();  // the shared buffer is free from here on
  wht_exchange<0>(v, sm, lane);
  // register i of lane l holds element k = R l + i, kept at position p = 32 i + l
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    wht_class<2, 5>(v, c);
#pragma unroll
    for (int i = c; i < 32; i += 4) sm[i * 32 + lane] = v[i];
  }
#endif
  fence_proxy_async_smem();
  __syncwarp();
  pre();
  if (lane == 0) {
    for (int b2 = 0; b2 < g.nb2; ++b2)
      for (int b0 = 0; b0 < g.nb0; ++b0)
        tma_store_4d(tmap, sm + (size_t)b2 * g.box2 * g.C + (size_t)b0 * (g.box0 / 2), b0 * g.box0, (int)rho,
                     b2 * g.box2, xcoord);
    bulk_commit();
  }
}

// Pass 2: tile of 2^HI rows x C = 2^(PB-HI) positions of one X-string's intermediate
// (one contiguous block); transform over the row bits, then per-lane moments.
template <int R, int HI, int QS, bool TM = false, typename V, typename Ready = NoHook>
__device__ __forceinline__ void p2_unit(const V *__restrict__ tile_ptr, V *sm, int lane, double *s,
                                        const QParams &qp, uint32_t ta = 0, const Ready &ready = Ready()) {
  (void)ta;
  constexpr int LOGR = ilog2c(R), PB = LOGR + 5, LOGC = PB - HI;
  static_assert(HI >= 1 && HI <= PB, "pass-2 bits out of range");
  V v[R];
#pragma unroll
  for (int i = 0; i < R; ++i) v[i] = __ldcg(tile_ptr + i * 32 + lane);
  if constexpr (LOGC >= 5) {
    reg_wht<R, LOGC - 5, LOGR>(v);
    ready();
#ifdef HM_TMEM_EXCHANGE
  } else if constexpr (TM && R == 32) {
    reg_wht<R, 0, LOGR>(v);
    ready();
    tmem_tile<HI>(v, ta);
    reg_wht<R, 0, 5 - LOGC>(v);
#endif
  } else {
    static_assert(R == 32, "32 values per lane");
#pragma unroll
    for (int b = 0; b < 8; ++b) wht_block<0, 2>(v, b);
    ready();
    wht_exchange<(LOGC < 2 ? LOGC : 2)>(v, sm, lane);
    if constexpr ((QS == QS_Q2 || (QS == QS_Q23 && sizeof(V) == 16)) && LOGC <= 3) {
      quad_moments<QS, LOGC>(v, s);
      return;
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) wht_class<(LOGC > 2 ? LOGC : 2), 5>(v, c);
  }
  lane_moments<R, QS>(v, s, qp, sm, lane);
}

}  // namespace hm
