// sre_wide.cuh -- exact-SRE transforms held by a group of G warps (G = 2, 4, 8): the whole
// transform of an X-string for n = 12, 13, 14 (2^(n-1) = 1024 G complex values) without
// leaving the SM.
//
// The WHT is real-linear, so the real and imaginary parts separate after the products:
//   phase A  lane l, register i of warp w holds the complex element e = 32 i + l + 1024 w:
//            the products f(e) and the butterflies over bits 5 .. 9 (32 complex registers);
//   exchange through the group's shared buffer, split into a real and an imaginary plane;
//   phase B  a lane holds 64 real values of one plane: bits 0 .. 4 and 10 in registers
//            (bit 0 inside a pair), so six bits run in registers instead of five, and for
//            G = 4, 8 bits 11 and 12 on lane bits, one shuffle and one FMA per value each.
// One shared-memory round trip per X-string (64 B per complex element on the L1 path with
// the two gathers; the lane levels of G = 4, 8 add 16 B each); the two-pass sweep it
// replaces at these sizes moved 144 B and went through L2 between its passes, a few stages
// of too few units.  Both precisions run 8 KB of planes per warp and value size, 8 (FP64,
// 255 registers) or 16 (FP32, 128 registers) warps per SM.  Measured on B200, whole sweep of
// the kernel, two-pass stages -> this (us):
//   q = 2   FP64  n = 12: 69 -> 31   n = 13: 226 -> 124   n = 14: 1107 -> 530
//           FP32  n = 12: 60 -> 32   n = 13: 144 -> 81    n = 14: 614 -> 308
//   n = 13, FP64: q = 2 and 3 231 -> 137, q = 4 724 -> 291, q = 2.5 1498 -> 1032
// FP64 at n = 13 is 1.04 clocks per complex element and SM, 0.55 of them FP64 issue.
#pragma once
#include "sre_kernels.cuh"

namespace hm {

// threads of one group meet (id 0 .. 15; the group's warps are whole warps)
template <int NT>
__device__ __forceinline__ void group_sync(int id) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(NT) : "memory");
}

// position of real element e of a plane in the group's buffer: 16-byte granules XOR-ed with
// bits 5 .. 7 of e, so that both the phase-A stores (lanes over bits 0 .. 4) and the phase-B
// loads (lanes over bits 5 .. 9, 16 bytes each) are free of bank conflicts
template <typename T>
__device__ __forceinline__ uint32_t wide_pos(uint32_t e) {
  constexpr int GS = sizeof(T) == 8 ? 1 : 2;  // log2 of the values per granule
  return e ^ (((e >> 5) & 7u) << GS);
}

// phase A's 32 complex registers -> the two planes
template <typename T, int G, typename V>
__device__ __forceinline__ void wide_put(const V (&v)[32], T *buf, int w, int lane) {
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    const uint32_t p = wide_pos<T>((uint32_t)(32 * i + lane)) + 1024u * w;
    buf[p] = v[i].x;
    buf[1024 * G + p] = v[i].y;
  }
}

// Element bits of a phase-B lane that are not in its registers: five on the lane number, the
// rest (with the plane as the top one) on the warp number.
//   G = 2: lanes 5 6 7 8 9,     warp: plane
//   G = 4: lanes 5 6 7 8 11,    warp: 9, plane
//   G = 8: lanes 5 6 7 11 12,   warp: 8, 9, plane
template <int G>
__device__ __forceinline__ uint32_t wide_base(int w, int lane) {
  if constexpr (G == 2) {
    return (uint32_t)lane << 5;
  } else if constexpr (G == 4) {
    return ((uint32_t)(lane & 15) << 5) | ((uint32_t)(lane >> 4) << 11) | ((uint32_t)(w & 1) << 9);
  } else {
    return ((uint32_t)(lane & 7) << 5) | ((uint32_t)(lane >> 3) << 11) | ((uint32_t)(w & 3) << 8);
  }
}

// the planes -> 32 pairs per lane: pair i holds bits 1 .. 4 = i & 15 and bit 10 = i >> 4, bit
// 0 inside the pair
template <typename T, int G, typename V>
__device__ __forceinline__ void wide_get(V (&v)[32], const T *buf, int w, int lane) {
  const T *plane = buf + (w >= G / 2 ? 1024 * G : 0);
  const uint32_t base = wide_base<G>(w, lane);
#pragma unroll
  for (int b = 0; b < 2; ++b) {
    if constexpr (sizeof(T) == 8) {
#pragma unroll
      for (int i = 0; i < 16; ++i)
        v[16 * b + i] = *reinterpret_cast<const V *>(plane + wide_pos<T>((base | (2 * i))) + 1024 * b);
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float4 q = *reinterpret_cast<const float4 *>(plane + wide_pos<T>((base | (4 * i))) + 1024 * b);
        v[16 * b + 2 * i] = make_float2(q.x, q.y);
        v[16 * b + 2 * i + 1] = make_float2(q.z, q.w);
      }
    }
  }
}

// one transform bit held by lane bit `m` (a mask): every value meets its partner's
template <typename V>
__device__ __forceinline__ void lane_wht(V (&v)[32], int lane, int m) {
  const float s = (lane & m) ? -1.0f : 1.0f;
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    const auto px = __shfl_xor_sync(0xffffffffu, v[i].x, m);
    const auto py = __shfl_xor_sync(0xffffffffu, v[i].y, m);
    v[i].x = fma(v[i].x, (decltype(px))s, px);
    v[i].y = fma(v[i].y, (decltype(py))s, py);
  }
}

// y^e for integer e >= 1 by repeated squaring, N values side by side
template <int N>
__device__ __forceinline__ void powi_many(const double (&y)[N], int e, double (&r)[N]) {
  double b[N];
#pragma unroll
  for (int t = 0; t < N; ++t) b[t] = y[t], r[t] = 1.0;
  while (e) {
    if (e & 1) {
#pragma unroll
      for (int t = 0; t < N; ++t) r[t] *= b[t];
    }
    e >>= 1;
    if (e) {
#pragma unroll
      for (int t = 0; t < N; ++t) b[t] *= b[t];
    }
  }
}

// Generic Renyi indices over the 64 values of a lane, staged in its own 64 slots of shared
// memory (sm[lane + 32 t]): a rolled loop of four values at a time, so that integer powers
// and pow() run four independent chains.
template <typename T>
__device__ __noinline__ void wide_moments_gen(const T *sm, int lane, double *s, const QParams &qp) {
  double a2 = 0.0, ag[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 1
  for (int t0 = 0; t0 < 64; t0 += 4) {
    double y[4], r[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const double f = (double)sm[lane + 32 * (t0 + t)];
      y[t] = f * f;
    }
    a2 += (y[0] + y[1]) + (y[2] + y[3]);
#pragma unroll 1
    for (int k = 0; k < qp.nq; ++k) {
      const double q = qp.q[k];
      if (q == floor(q) && q >= 1.0 && q <= 16.0) {
        powi_many<4>(y, (int)q, r);
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

// Butterflies of phase B's register bits and the per-lane sums of F^2 and (F^2)^q.
// q = 2 alone: the last two bits are not transformed.  For four values u_e before them,
// with c_d = sum_e u_e u_(e^d), the four outputs satisfy sum F^2 = 4 c_0 and
// sum F^4 = 4 (c_0^2 + c_1^2 + c_2^2 + c_3^2) (F_k^2 = sum_d (-1)^(k.d) c_d, Parseval over k):
// 15 operations for the four values instead of 8 for the two bits and 12 for the powers.
template <int QS, typename T, typename V>
__device__ __forceinline__ void wide_moments(V (&v)[32], double *s, const QParams &qp, T *sm, int lane) {
  if constexpr (QS == QS_Q2) {
    reg_wht<32, 0, 4>(v);
    double a2[2] = {0.0, 0.0}, m0[2] = {0.0, 0.0}, h1 = 0.0, h2 = 0.0, h3 = 0.0;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const double u0 = v[i].x, u1 = v[i].y, u2 = v[i + 16].x, u3 = v[i + 16].y;
      const double c0 = fma(u0, u0, fma(u1, u1, fma(u2, u2, u3 * u3)));
      const double c1 = fma(u0, u1, u2 * u3), c2 = fma(u0, u2, u1 * u3), c3 = fma(u0, u3, u1 * u2);
      a2[i & 1] += c0;
      m0[i & 1] = fma(c0, c0, m0[i & 1]);
      h1 = fma(c1, c1, h1);
      h2 = fma(c2, c2, h2);
      h3 = fma(c3, c3, h3);
    }
    s[0] = 4.0 * (a2[0] + a2[1]);
    s[1] = 4.0 * ((m0[0] + m0[1]) + 4.0 * ((h1 + h2) + h3));
  } else {
    reg_wht<32, 0, 5>(v);
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      const auto a = v[i].x, b = v[i].y;
      v[i].x = a + b;
      v[i].y = a - b;
    }
    if constexpr (QS == QS_GEN) {
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        sm[lane + 64 * i] = v[i].x;
        sm[lane + 64 * i + 32] = v[i].y;
      }
      wide_moments_gen(sm, lane, s, qp);
    } else {
      lane_moments<32, QS>(v, s, qp, (V *)nullptr, lane);  // q = 2 and 3: no staging
    }
  }
}

// Groups per SM: FP64 8 warps (255 registers), FP32 16 warps (128 registers).
template <typename T, int G> struct WideOcc { static constexpr int value = (sizeof(T) == 8 ? 8 : 16) / G; };

// n = 11 + log2 G: one CTA of G warps per X-string at a time, X-strings strided over the grid
template <typename T, int G, int QS>
__global__ void __launch_bounds__(32 * G, WideOcc<T, G>::value) k_sre_wide(SreArgs a) {
  using V = typename VT<T>::V;
  constexpr int NB = 10 + ilog2c(G), NQ = QSet<QS>::NQ;  // bits of the half transform
  extern __shared__ __align__(128) unsigned char smem_wide[];
  T *buf = reinterpret_cast<T *>(smem_wide);  // two planes of 1024 G values
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const V *psi = reinterpret_cast<const V *>(a.psi);
  const uint32_t e0 = 1024u * w + lane;
  dd acc[NQ + 1];
#pragma unroll
  for (int t = 0; t <= NQ; ++t) acc[t] = dd{0.0, 0.0};
  for (uint64_t k = a.k_begin + blockIdx.x; k < a.k_end; k += gridDim.x) {
    const uint32_t x = (uint32_t)gray_code(k);
    V v[32];
    if (x != 0) {
      // r = e with a zero inserted at the highest set bit of x: e + (the bits from there up)
      const uint32_t up = ~((1u << (31 - __clz((int)x))) - 1u);
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        const uint32_t e = e0 + 32u * i, r = e + (e & up);
        v[i] = conj_mul(ld_psi(psi + r), ld_psi(psi + (r ^ x)));
      }
    } else {
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        const uint32_t e = e0 + 32u * i;
        v[i] = zero_pair(ld_psi(psi + e), ld_psi(psi + e + (1u << NB)));
      }
    }
    reg_wht<32, 0, 5>(v);  // element bits 5 .. 9
    __syncthreads();       // the previous X-string's values have been read
    wide_put<T, G>(v, buf, w, lane);
    __syncthreads();
    wide_get<T, G>(v, buf, w, lane);
    if constexpr (G == 4) lane_wht(v, lane, 16);
    if constexpr (G == 8) {
      lane_wht(v, lane, 8);
      lane_wht(v, lane, 16);
    }
    double s[NQ + 1];
    if constexpr (QS == QS_GEN) __syncthreads();  // the moments stage their values in the buffer
    wide_moments<QS>(v, s, a.qp, buf + 2048 * w, lane);
    s[0] = x == 0 ? s[0] : 4.0 * s[0];
#pragma unroll
    for (int t = 0; t < NQ; ++t) s[1 + t] *= q_scale<QS>(t, x == 0, a.qp);
#pragma unroll
    for (int t = 0; t <= NQ; ++t) dd_add(acc[t], s[t]);
  }
  // fixed-order butterfly reduction of the lanes' accumulators
#pragma unroll
  for (int t = 0; t <= NQ; ++t) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      dd other;
      other.hi = __shfl_xor_sync(0xffffffffu, acc[t].hi, o);
      other.lo = __shfl_xor_sync(0xffffffffu, acc[t].lo, o);
      dd_add_dd(acc[t], other);
    }
  }
  if (lane == 0) write_partials<NQ>(a.partials, blockIdx.x * G + w, acc);
}

}  // namespace hm
