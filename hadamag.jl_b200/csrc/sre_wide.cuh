// sre_wide.cuh -- exact-SRE transforms held by a group of G warps (G = 2, 4, 8; in FP64 also
// 1, in FP32 also 16): the whole transform of an X-string for n = 12, 13, 14 (FP64 also 11,
// FP32 15; 2^(n-1) = 1024 G complex values) without leaving the SM, and the two-pass sweep
// of larger n.
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
//                 n = 15: 2180 -> 1430 (2030 with the two-pass sweep below)
//   n = 13, FP64: q = 2 and 3 231 -> 136, q = 4 724 -> 149, q = 2.5 1498 -> 151
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
// bits 5 .. 7 of e (G = 16: bits 5, 6 and 11), the low three bits of the phase-B lane, so
// that both the phase-A stores (lanes over bits 0 .. 4) and the phase-B loads (16 bytes a
// lane) are free of bank conflicts
template <typename T, int G>
__device__ __forceinline__ uint32_t wide_pos(uint32_t e) {
  constexpr int GS = sizeof(T) == 8 ? 1 : 2;  // log2 of the values per granule
  const uint32_t f = G == 16 ? ((e >> 5) & 3u) | ((e >> 9) & 4u) : (e >> 5) & 7u;
  return e ^ (f << GS);
}

// phase A's 32 complex registers -> the two planes
template <typename T, int G, typename V>
__device__ __forceinline__ void wide_put(V (&v)[32], T *buf, int w, int lane) {
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    wht_class<2, 5>(v, c);
#pragma unroll
    for (int i = c; i < 32; i += 4) {
      const uint32_t p = wide_pos<T, G>((uint32_t)(32 * i + lane) + 1024u * w);
      buf[p] = v[i].x;
      buf[1024 * G + p] = v[i].y;
    }
  }
}

// Element bits of a phase-B lane that are not in its registers: five on the lane number, the
// rest (with the plane as the top one) on the warp number.
//   G = 1: lanes 5 6 7 8 9,     the plane in the registers, where larger G have bit 10
//   G = 2: lanes 5 6 7 8 9,     warp: plane
//   G = 4: lanes 5 6 7 8 11,    warp: 9, plane
//   G = 8: lanes 5 6 7 11 12,   warp: 8, 9, plane
//   G = 16: lanes 5 6 11 12 13, warp: 7, 8, 9, plane
template <int G>
__device__ __forceinline__ uint32_t wide_base(int w, int lane) {
  if constexpr (G <= 2) {
    return (uint32_t)lane << 5;
  } else if constexpr (G == 4) {
    return ((uint32_t)(lane & 15) << 5) | ((uint32_t)(lane >> 4) << 11) | ((uint32_t)(w & 1) << 9);
  } else if constexpr (G == 8) {
    return ((uint32_t)(lane & 7) << 5) | ((uint32_t)(lane >> 3) << 11) | ((uint32_t)(w & 3) << 8);
  } else {
    return ((uint32_t)(lane & 3) << 5) | ((uint32_t)(lane >> 2) << 11) | ((uint32_t)(w & 7) << 7);
  }
}

// the planes -> 32 pairs per lane: pair i holds bits 1 .. 4 = i & 15 and bit 10 = i >> 4, bit
// 0 inside the pair
template <typename T, int G, typename V>
__device__ __forceinline__ void wide_get(V (&v)[32], const T *buf, int w, int lane) {
  const T *plane = buf + (G > 1 && w >= G / 2 ? 1024 * G : 0);
  const uint32_t base = wide_base<G>(w, lane);
#pragma unroll
  for (int b = 0; b < 2; ++b) {
    if constexpr (sizeof(T) == 8) {
#pragma unroll
      for (int i = 0; i < 16; ++i)
        v[16 * b + i] = *reinterpret_cast<const V *>(plane + wide_pos<T, G>(base | (2 * i)) + 1024 * b);
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float4 q = *reinterpret_cast<const float4 *>(plane + wide_pos<T, G>(base | (4 * i)) + 1024 * b);
        v[16 * b + 2 * i] = make_float2(q.x, q.y);
        v[16 * b + 2 * i + 1] = make_float2(q.z, q.w);
      }
    }
  }
}

// wide_get and wide_put the other way, for a backward transform: phase B's values into the
// planes (each lane's own addresses), and the planes into phase A's registers with the
// butterflies over bits 5 .. 9
template <typename T, int G, typename V>
__device__ __forceinline__ void wide_unget(const V (&v)[32], T *buf, int w, int lane) {
  static_assert(sizeof(T) == 8, "FP64 only");
  T *plane = buf + (G > 1 && w >= G / 2 ? 1024 * G : 0);
  const uint32_t base = wide_base<G>(w, lane);
#pragma unroll
  for (int b = 0; b < 2; ++b)
#pragma unroll
    for (int i = 0; i < 16; ++i)
      *reinterpret_cast<V *>(plane + wide_pos<T, G>(base | (2 * i)) + 1024 * b) = v[16 * b + i];
}
template <typename T, int G, typename V>
__device__ __forceinline__ void wide_unput(V (&v)[32], const T *buf, int w, int lane) {
#pragma unroll
  for (int b = 0; b < 8; ++b) {
#pragma unroll
    for (int i = 4 * b; i < 4 * b + 4; ++i) {
      const uint32_t p = wide_pos<T, G>((uint32_t)(32 * i + lane) + 1024u * w);
      v[i].x = buf[p];
      v[i].y = buf[1024 * G + p];
    }
    wht_block<0, 2>(v, b);
  }
#pragma unroll
  for (int c = 0; c < 4; ++c) wht_class<2, 5>(v, c);
}

// Butterflies over the LV low bits of the register index (and, with PAIR, over the bit inside
// a pair), then the per-lane sums of F^2 and (F^2)^q.
// q = 2 and, in FP64, q = 2 and 3: the last two bits are not transformed (QuadSums, CubeSums;
// in FP32 the two levels are cheap and the cubes would cost as many FP64 operations as the
// powers).
template <int QS, int LV, bool PAIR, typename T, typename V>
__device__ __forceinline__ void wide_moments(V (&v)[32], double *s, const QParams &qp, T *sm, int lane) {
  if constexpr (QS == QS_Q2 || (QS == QS_Q23 && sizeof(T) == 8)) {
    constexpr int TOP = PAIR ? LV - 1 : LV - 2;  // transformed explicitly: index bits 0 .. TOP-1
#pragma unroll
    for (int b = 0; b < 8; ++b) wht_block<0, TOP>(v, b);
    LevelSums<QS> quad;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      wht_class<0, TOP>(v, c);
#pragma unroll
      for (int i = TOP >= 2 ? c : 8 * c; i < (TOP >= 2 ? 32 : 8 * c + 8); i += (TOP >= 2 ? 4 : 1)) {
        if constexpr (PAIR) {
          if ((i >> TOP) & 1) continue;
          const int k = i | (1 << TOP);
          quad.add(i & 1, v[i].x, v[i].y, v[k].x, v[k].y);
        } else {
          if ((i >> TOP) & 3) continue;
          const int k = i | (1 << TOP), m = i | (2 << TOP);
          quad.add(0, v[i].x, v[k].x, v[m].x, v[m | k].x);
          quad.add(1, v[i].y, v[k].y, v[m].y, v[m | k].y);
        }
      }
    }
    quad.get(s);
  } else {
    reg_wht<32, 0, LV>(v);
    if constexpr (PAIR) {
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        const auto a = v[i].x, b = v[i].y;
        v[i].x = a + b;
        v[i].y = a - b;
      }
    }
    lane_moments<32, QS>(v, s, qp, reinterpret_cast<V *>(sm), lane);
  }
}

// Phase A of X-string x for element e0 + 32 i in register i (e0 includes the lane): products
// and butterflies over bits 5 .. 9.  r(e) is e with a zero inserted at the highest set bit
// of x, e + (the bits of e from there up), for any position of that bit; x = 0 pairs the
// top bit (half = 2^(n-1)).
template <typename V>
__device__ __forceinline__ void wide_build(V (&v)[32], const V *__restrict__ psi, uint32_t x, uint32_t e0,
                                           uint32_t half) {
  if (x != 0) {
    const uint32_t up = ~((1u << (31 - __clz((int)x))) - 1u);
#pragma unroll
    for (int b = 0; b < 8; ++b) {
#pragma unroll
      for (int i = 4 * b; i < 4 * b + 4; ++i) {
        const uint32_t e = e0 + 32u * i, r = e + (e & up);
        v[i] = conj_mul(ld_psi(psi + r), ld_psi(psi + (r ^ x)));
      }
      wht_block<0, 2>(v, b);
    }
  } else {
#pragma unroll
    for (int b = 0; b < 8; ++b) {
#pragma unroll
      for (int i = 4 * b; i < 4 * b + 4; ++i) {
        const uint32_t e = e0 + 32u * i;
        v[i] = zero_pair(ld_psi(psi + e), ld_psi(psi + e + half));
      }
      wht_block<0, 2>(v, b);
    }
  }
}

// the transform bits that phase B keeps on lane bits
template <int G, typename V>
__device__ __forceinline__ void wide_lane_bits(V (&v)[32], int lane) {
  if constexpr (G == 4) lane_wht(v, lane, 16);
  if constexpr (G == 8) {
    lane_wht(v, lane, 8);
    lane_wht(v, lane, 16);
  }
  if constexpr (G == 16) {
    lane_wht(v, lane, 4);
    lane_wht(v, lane, 8);
    lane_wht(v, lane, 16);
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
    wide_build(v, psi, x, e0, 1u << NB);
    __syncthreads();       // the previous X-string's values have been read
    wide_put<T, G>(v, buf, w, lane);
    __syncthreads();
    wide_get<T, G>(v, buf, w, lane);
    wide_lane_bits<G>(v, lane);
    double s[NQ + 1];
    if (QS == QS_GEN && !a.qp.direct) __syncthreads();  // the moments stage their values in the buffer
    wide_moments<QS, (G > 1 ? 5 : 4), true>(v, s, a.qp, buf + 2048 * w, lane);
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
  fold_last<NQ, 32 * G>(a, (int)gridDim.x * G);
}

// ---------------------------------------------------------------------------------
// Two-pass sweep for 15 <= n <= 21 as a sequence of stage kernels (chained and replayed as
// k_sre_stage's: stage t runs pass 1 of batch t and pass 2 of batch t - 1, slot b & 1).
//   pass 1  a group of G warps transforms the low 10 + log2 G bits of the (n-1)-bit index:
//           phase A, exchange, phase B as above.  Its 2048 G real values leave straight from
//           the registers as one row of the intermediate, pairs in register order (any
//           fixed relabelling of the columns is invisible to the sums): whole 512-byte
//           (FP64) or 256-byte stores, no staging.
//   pass 2  columns of the 2^HI rows, HI = n - 11 - log2 G.  A lane holds 64 values; a warp
//           2^HI rows of 2^(11-HI) columns.  HI <= 5: pairs of columns, up to 32 rows in
//           registers.  HI >= 6: six row bits in registers, the others on lane bits.
// No value crosses shared memory in pass 2.  L1-path bytes per complex element: 32 gather,
// 32 exchange, 16 store, 16 load, 16 per lane bit, against 144 for rows and tiles of 1024
// with an exchange in each pass and tensor stores.
struct WideArgs {
  const void *psi;
  void *ring;       // 2 slots x X strings x 2^n values of T: rows of 2048 G
  double *slots;    // per warp: 2 (1 + NQ) doubles
  unsigned *stage;  // [0] stage index of node 0 of the current graph replay
  uint64_t k_begin, k_end;
  QParams qp;
  int X, nbatch;
  int node;         // position of this launch in the captured graph
};

template <int G> struct WideCta { static constexpr int WARPS = G < 4 ? 4 : G; };

template <typename T, int G, int HI, int QS>
__global__ void __launch_bounds__(32 * WideCta<G>::WARPS, (sizeof(T) == 8 ? 8 : 16) / WideCta<G>::WARPS)
    k_sre_wide_stage(const __grid_constant__ WideArgs a) {
  using V = typename VT<T>::V;
  constexpr int NQ = QSet<QS>::NQ, NG = WideCta<G>::WARPS / G;  // groups per CTA
  constexpr uint32_t ROW = 2048 * G, NROW = 1u << HI;
  extern __shared__ __align__(128) unsigned char smem_wide[];
  allow_next_grid();
  // the base only changes between replays, after every node of the replay has finished
  const long long t = (long long)*(volatile unsigned *)a.stage + a.node;
  // padding stages of the last graph replay end after the stage that they follow (see k_sre_stage)
  if (t > a.nbatch) {
    wait_prior_grid();
    return;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int grp = warp / G, w = warp % G;
  T *buf = reinterpret_cast<T *>(smem_wide) + (size_t)grp * ROW;
  const V *psi = reinterpret_cast<const V *>(a.psi);
  T *ring = reinterpret_cast<T *>(a.ring);
  const long long per = (long long)a.X * NROW;    // items (row or G column blocks) per pass
  const long long n1 = t < a.nbatch ? per : 0;    // pass 1 of batch t
  constexpr uint32_t CHUNK = (2048u >> HI) * sizeof(T);    // bytes of a unit in each row
  constexpr uint32_t UPI = CHUNK < 128 ? 128 / CHUNK : 1;  // units per item: whole L2 lines
  const long long n2 = t >= 1 ? per / UPI : 0;             // pass 2 of batch t - 1
  const long long gid = (long long)blockIdx.x * NG + grp, ngrp = (long long)gridDim.x * NG;
  dd acc[NQ + 1];
#pragma unroll
  for (int q = 0; q <= NQ; ++q) acc[q] = dd{0.0, 0.0};
  // One pass-1 item first (its gathers and butterflies overlap the previous stage's tail), then
  // the pass-2 items (the previous stage's rows are still in L2), then the rest of pass 1.
  const long long nfirst = n1 < ngrp ? n1 : ngrp;
  for (long long u = gid; u < n1 + n2; u += ngrp) {
    const bool p2 = u >= nfirst && u < nfirst + n2;
    const long long r = p2 ? u - nfirst : (u < nfirst ? u : u - n2);
    const long long b = p2 ? t - 1 : t;
    const uint32_t xs = (uint32_t)(r % a.X), sub = (uint32_t)(r / a.X);
    const uint64_t k = a.k_begin + (uint64_t)b * a.X + xs;
    if (k >= a.k_end) continue;
    const uint32_t x = (uint32_t)gray_code(k);
    T *inter = ring + ((size_t)(b & 1) * a.X + xs) * ((size_t)NROW * ROW);
    V v[32];
    if (!p2) {
      wide_build(v, psi, x, sub * (1024u * G) + 1024u * w + lane, NROW * (1024u * G));
      group_sync<32 * G>(1 + grp);  // the group's previous values have been read
      wide_put<T, G>(v, buf, w, lane);
      group_sync<32 * G>(1 + grp);
      wide_get<T, G>(v, buf, w, lane);
      wide_lane_bits<G>(v, lane);
#pragma unroll
      for (int b = 0; b < 8; ++b) wht_block<0, 2>(v, b);
      wait_prior_grid();  // the slot that the previous stage's pass 2 read
      V *row = reinterpret_cast<V *>(inter + (size_t)sub * ROW) + 1024 * w + lane;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        wht_class<2, 5>(v, c);
#pragma unroll
        for (int i = c; i < 32; i += 4) {
          const auto p = v[i].x, q = v[i].y;
          v[i].x = p + q;
          v[i].y = p - q;
          __stcg(row + 32 * i, v[i]);
        }
      }
    } else {
      wait_prior_grid();  // the previous stage's rows
#pragma unroll 1
      for (uint32_t h = 0; h < UPI; ++h) {
        const uint32_t unit = (sub * G + w) * UPI + h;  // block of 2^(11-HI) columns
        const T *col = inter + ((size_t)unit << (11 - HI));
        double s[NQ + 1];
        if constexpr (HI <= 5) {
          // register i: row i mod 2^HI, column block i >> HI of 64 columns (a pair per lane)
#pragma unroll
          for (int i = 0; i < 32; ++i)
            v[i] = __ldcg(reinterpret_cast<const V *>(col + (size_t)(i & (NROW - 1)) * ROW + 64 * (i >> HI)) + lane);
        } else {
          // lane: column in its low 11 - HI bits, the row's low HI - 6 bits above them;
          // register pair i: rows with bits HI-6 = (x, y) and i above
          constexpr int CB = 11 - HI, LB = HI - 6;
          const T *p = col + (lane & ((1 << CB) - 1)) + (size_t)(lane >> CB) * ROW;
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            v[i].x = __ldcg(p + (size_t)((2 * i) << LB) * ROW);
            v[i].y = __ldcg(p + (size_t)((2 * i + 1) << LB) * ROW);
          }
#pragma unroll
          for (int m = 1 << CB; m < 32; m <<= 1) lane_wht(v, lane, m);
        }
        if (QS == QS_GEN && !a.qp.direct) group_sync<32 * G>(1 + grp);  // the moments stage in the buffer
        wide_moments<QS, (HI <= 5 ? HI : 5), (HI > 5)>(v, s, a.qp, buf + 2048 * w, lane);
        s[0] = x == 0 ? s[0] : 4.0 * s[0];
#pragma unroll
        for (int q = 0; q < NQ; ++q) s[1 + q] *= q_scale<QS>(q, x == 0, a.qp);
#pragma unroll
        for (int q = 0; q <= NQ; ++q) dd_add(acc[q], s[q]);
      }
      // The columns are dead once read (pass 1 of the next stage rewrites their slot, after its
      // griddepcontrol.wait on this launch): drop their L2 lines without writing them back.
      constexpr uint32_t LPR = CHUNK * UPI / 128;  // lines per row
      const T *line = inter + ((size_t)((sub * G + w) * UPI) << (11 - HI));
      __syncwarp();  // every lane's reads come before
#pragma unroll
      for (uint32_t ln = lane; ln < NROW * LPR; ln += 32)
        asm volatile("discard.global.L2 [%0], 128;" ::"l"(reinterpret_cast<const char *>(
                         line + (size_t)(ln / LPR) * ROW) + (ln % LPR) * 128)
                     : "memory");
    }
  }
  if (n2 > 0) {
    // fixed-order butterfly reduction of the lanes' accumulators
#pragma unroll
    for (int q = 0; q <= NQ; ++q) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        dd other;
        other.hi = __shfl_xor_sync(0xffffffffu, acc[q].hi, o);
        other.lo = __shfl_xor_sync(0xffffffffu, acc[q].lo, o);
        dd_add_dd(acc[q], other);
      }
    }
    if (lane == 0) {
      wait_prior_grid();  // the previous stage updates the same slot
      double *sl = a.slots + ((size_t)blockIdx.x * WideCta<G>::WARPS + warp) * 2 * (NQ + 1);
#pragma unroll
      for (int q = 0; q <= NQ; ++q) {
        dd d{sl[2 * q], sl[2 * q + 1]};
        dd_add_dd(d, acc[q]);
        sl[2 * q] = d.hi;
        sl[2 * q + 1] = d.lo;
      }
    }
  }
}

}  // namespace hm
