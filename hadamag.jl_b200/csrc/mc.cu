// mc.cu -- MC_SRE: Metropolis chains over X-strings (src/SRE.jl:110-192,
// src/Backends/Threads.jl:161-221, Simpson of src/Helpers.jl:223-236).
//
// Few qubits or few chains (see one_launch): one launch runs whole chains, each inside one
// warp, one CTA or one cluster of CTAs, with no exchange between chains.  Otherwise all
// chains advance together: a step evaluates m(x) and p2(x) of every chain's proposal with
// a pass-1 and a pass-2 kernel over (chain, row / tile) units, then one update kernel
// applies the acceptance rule of src/SRE.jl:172-186 on the device and forms the next
// proposal from the injected stream.  Kernel arguments do not change between steps (the
// step counter lives in device memory), so a block of steps is captured once as a CUDA
// graph and replayed.
#include <math.h>

#include <utility>
#include <vector>

#include "hm_ctx.h"
#include "sre_wide.cuh"

namespace hm {

namespace {

struct Chain {
  uint64_t cur, prop;  // current X-string, proposal under evaluation
  double prob, m2, p2; // currPROB, currM2, currP2
  double sM2, sM2sq, sP2;
  double beta;
  long long n;
};

struct McArgs {
  const double2 *psi;
  const double2 *psi_sw[16];  // two-pass relabelled copies
  double2 *inter;             // nbeta x 2^(n-1)
  double *part;               // nbeta x U x 2 (p2, m) per pass-2 tile
  Chain *ch;
  const uint64_t *pd;  // nbeta x nsamples
  const double *rs;
  long long *step;  // device step counter
  unsigned *upd_done;  // blocks of k_mc_update that finished the current step
  QParams qp;
  int n, nbeta, nsamples, U;  // nbeta: chains of this run
  int chain0, nbeta_grid;     // first chain's index in the beta grid of nbeta_grid points
  double p2_0, m0;  // x = 0 sample
};

// q = 2 or generic through QS_GEN
template <int QS>
__device__ __forceinline__ double moment_scale(const QParams &qp) {
  return QS == QS_Q2 ? 16.0 : qp.scale[0];
}

// n >= 16, pass 1: warp units (chain, row)
template <int HI>
__global__ void __launch_bounds__(128) k_mc_p1(McArgs a) {
  constexpr int R = 32, PB = 10;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double2 *sm = reinterpret_cast<double2 *>(smraw) + warp * 32 * R;
  allow_next_grid();
  wait_prior_grid();  // the previous update has written the proposals
  if (*a.step >= a.nsamples) return;
  const long long u = (long long)blockIdx.x * 4 + warp;
  if (u >= (long long)a.nbeta * a.U) return;
  const int c = (int)(u / a.U);
  const uint64_t row = (uint64_t)(u % a.U);
  const uint64_t x = a.ch[c].prop;
  if (x == 0) return;
  XInfo xx;
  xx.active = 1;
  xx.sw = -1;
  xx.xt = x;
  xx.jt = 63 - __clzll((long long)x);
  if (xx.jt < PB) {
    xx.sw = xx.jt;
    xx.xt = (x ^ (1ull << xx.jt)) | (1ull << (a.n - 1));
    xx.jt = a.n - 1;
  }
  const double2 *src = xx.sw < 0 ? a.psi : a.psi_sw[xx.sw];
  p1_unit<R, HI>(src, xx, row, a.inter + (size_t)c * ((size_t)1 << (a.n - 1)), sm, lane);
}

// n >= 16, pass 2: warp units (chain, tile) -> part[chain][tile].  Three CTAs per SM: left to
// itself the compiler gives the generic q 198 registers, which leaves two and idle time in the
// powers (q = 2.7, us per step: n = 18, 13 chains 87 -> 63; n = 16, 201 chains 265 -> 213).
template <int HI, int QS>
__global__ void __launch_bounds__(128, 3) k_mc_p2(McArgs a) {
  constexpr int R = 32, PB = 10;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double2 *sm = reinterpret_cast<double2 *>(smraw) + warp * 32 * R;
  allow_next_grid();
  wait_prior_grid();  // pass 1 of this step has stored the rows
  if (*a.step >= a.nsamples) return;
  const long long u = (long long)blockIdx.x * 4 + warp;
  if (u >= (long long)a.nbeta * a.U) return;
  const int c = (int)(u / a.U);
  const uint64_t tile = (uint64_t)(u % a.U);
  if (a.ch[c].prop == 0) return;
  double s[5];
  p2_unit<R, HI, QS>(a.inter + (size_t)c * ((size_t)1 << (a.n - 1)) + (tile << PB), sm, lane, s, a.qp);
  const double p2 = warp_sum(s[0]) * 4.0, m = warp_sum(s[1]) * moment_scale<QS>(a.qp);
  if (lane == 0) {
    a.part[2 * u] = p2;
    a.part[2 * u + 1] = m;
  }
}

// Metropolis update of every chain (src/SRE.jl:164-186) and next proposal.  One warp per
// chain, MC_UPD_WARPS chains per block, as many blocks as the chains need:
// the warp's lanes fold the chain's per-tile partials (lane l takes tiles l, l + 32, ...
// in double-double, then a fixed butterfly; the order never changes), and lane 0 updates
// the chain.  The last block to finish advances the device step counter (a ticket taken
// with an atomic after a fence, so every block has read the counter before it moves;
// nothing waits).
constexpr int MC_UPD_WARPS = 4;
__global__ void __launch_bounds__(MC_UPD_WARPS * 32) k_mc_update(McArgs a) {
  allow_next_grid();
  wait_prior_grid();  // this step's evaluation has finished
  const long long t = *a.step;
  const int c = blockIdx.x * MC_UPD_WARPS + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (t < a.nsamples && c < a.nbeta) {
    Chain ch = a.ch[c];
    const uint64_t prop = ch.prop;
    double m_prop = 0.0, p2_prop = 0.0;
    if (prop != 0) {
      dd sp{0.0, 0.0}, sm{0.0, 0.0};
      for (int i = lane; i < a.U; i += 32) {
        dd_add(sp, a.part[2 * ((size_t)c * a.U + i)]);
        dd_add(sm, a.part[2 * ((size_t)c * a.U + i) + 1]);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        dd op, om;
        op.hi = __shfl_xor_sync(0xffffffffu, sp.hi, o);
        op.lo = __shfl_xor_sync(0xffffffffu, sp.lo, o);
        om.hi = __shfl_xor_sync(0xffffffffu, sm.hi, o);
        om.lo = __shfl_xor_sync(0xffffffffu, sm.lo, o);
        dd_add_dd(sp, op);
        dd_add_dd(sm, om);
      }
      p2_prop = sp.hi + sp.lo;
      m_prop = sm.hi + sm.lo;
    }
    if (lane == 0) {
      p2_prop /= (double)(1ull << a.n);
      const double pb = pow(m_prop, ch.beta);
      const double r = a.rs[(size_t)c * a.nsamples + t];
      if ((r < pb / ch.prob) && (prop != 0)) {
        ch.cur = prop;
        ch.prob = pb;
        ch.m2 = -log2(m_prop);
        ch.p2 = p2_prop;
      }
      ch.sM2 += ch.m2;
      ch.sM2sq += ch.m2 * ch.m2;
      ch.sP2 += ch.p2;
      ch.n += 1;
      if (t + 1 < a.nsamples) ch.prop = ch.cur ^ a.pd[(size_t)c * a.nsamples + t + 1];
      a.ch[c] = ch;
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    const unsigned ticket = atomicAdd(a.upd_done, 1u);
    if (ticket == gridDim.x - 1) {
      *a.upd_done = 0;
      if (t < a.nsamples) *a.step = t + 1;
    }
  }
}

// ---------------------------------------------------------------------------------
// n <= 17: one launch runs every step of every chain.  A chain never needs another one, so
// a chain belongs to one CTA or one cluster of CTAs for the whole run, its state stays in
// registers, and a step costs barriers of that CTA or cluster instead of two or three
// launches (about 4 us each way at 13 chains, whose 416 units at n = 16 also left most of
// the GPU idle in each of them).  What bounds a step is its serial chain: two gathers from
// L2, two exchanges, the sums, pow().  Figures at one_launch in run_mc.
struct McChain {
  uint64_t cur = 0, prop = 0;
  double prob = 1e-120, m2 = 0.0, p2 = 0.0, sM2 = 0.0, sM2sq = 0.0, sP2 = 0.0, beta = 0.0;
  const uint64_t *pd;
  const double *rs;
  double r;         // uniform of the current step
  uint64_t pd_next;  // flips of the next step, loaded a step ahead

  __device__ __forceinline__ void start(const McArgs &a, int c) {
    beta = (double)(a.chain0 + c) / (double)(a.nbeta_grid - 1);
    p2 = a.p2_0;
    pd = a.pd + (size_t)c * a.nsamples;
    rs = a.rs + (size_t)c * a.nsamples;
    prop = pd[0];
  }
  // loads whose latency the evaluation hides
  __device__ __forceinline__ void fetch(const McArgs &a, int t) {
    r = rs[t];
    pd_next = t + 1 < a.nsamples ? pd[t + 1] : 0;
  }
  // the acceptance rule of src/SRE.jl:172-186 and the next proposal
  __device__ __forceinline__ void step(const McArgs &a, double p2_prop, double m_prop) {
    const double pb = pow(m_prop, beta);
    if ((r < pb / prob) && (prop != 0)) {
      cur = prop;
      prob = pb;
      m2 = -log2(m_prop);
      p2 = p2_prop / (double)(1ull << a.n);
    }
    sM2 += m2;
    sM2sq += m2 * m2;
    sP2 += p2;
    prop = cur ^ pd_next;
  }
  __device__ __forceinline__ void finish(const McArgs &a, int c) const {
    Chain ch;
    ch.cur = cur;
    ch.prop = prop;
    ch.prob = prob;
    ch.m2 = m2;
    ch.p2 = p2;
    ch.sM2 = sM2;
    ch.sM2sq = sM2sq;
    ch.sP2 = sP2;
    ch.beta = beta;
    ch.n = a.nsamples;
    a.ch[c] = ch;
  }
};

// n <= 11: one warp per chain
template <int NB, int QS>
__global__ void __launch_bounds__(32) k_mc_chain_warp(McArgs a) {
  constexpr int R = 32;
  extern __shared__ __align__(16) unsigned char smraw[];
  double2 *sm = reinterpret_cast<double2 *>(smraw);
  const int c = blockIdx.x, lane = threadIdx.x;
  McChain ch;
  ch.start(a, c);
  for (int t = 0; t < a.nsamples; ++t) {
    ch.fetch(a, t);
    double p2 = 0.0, m = 0.0;
    if (ch.prop != 0) {  // a zero proposal is never accepted; its moments are not used
      const uint32_t x = (uint32_t)ch.prop, up = ~((1u << (31 - __clz((int)x))) - 1u);
      double2 v[R];
#pragma unroll
      for (int i = 0; i < R; ++i) {
        const uint32_t e = (uint32_t)(i * 32 + lane);
        double2 f = make_double2(0.0, 0.0);
        if (i * 32 < (1 << NB) && e < (1u << NB)) {
          const uint32_t r = e + (e & up);
          f = conj_mul(__ldg(a.psi + r), __ldg(a.psi + (r ^ x)));
        }
        v[i] = f;
      }
      if constexpr (NB > 5) reg_wht<R, 0, NB - 5>(v);
      transpose_ab<R>(v, sm, lane);
      reg_wht<R, 0, (NB < 5 ? NB : 5)>(v);
      double s[5];
      lane_moments<R, QS>(v, s, a.qp, sm, lane);
      p2 = warp_sum(s[0]) * 4.0;
      m = warp_sum(s[1]) * moment_scale<QS>(a.qp);
    }
    ch.step(a, p2, m);
  }
  if (lane == 0) ch.finish(a, c);
}

// n = 11 + L, 1 <= L <= 6: the 2^L warps of a chain, W to a CTA and CS CTAs to a cluster, hold
// its 2^(n-1) complex elements: phase A of sre_wide.cuh with the warp number as element
// bits 10 .. 9 + L, and the exchange through the cluster's shared memory into the warp that
// runs phase B.  There, warps take the plane and the top L - 1 of bits 5 .. 9, lanes bits
// 11 .. 9 + L (low lane bits) and the rest of 5 .. 9, registers bits 0 .. 4 and 10.
//   position of a value in its phase-B warp's 2048: [source warp][its bits 5 .. 10-L][bits 0 .. 4],
//   16-byte granules XOR-ed with the reading lane's low three bits (no bank conflicts).
// Bits 11 and up then run on a lane bit (L = 2) or, L >= 3, in registers after a transpose
// of the warp's own slice.  A step has two barriers: the values have arrived; the warps'
// sums have.  Every warp adds up all sums in the same order and takes the same decision.
template <int CS>
__device__ __forceinline__ void chain_sync() {
  if constexpr (CS == 1) {
    __syncthreads();
  } else {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
}
template <int CS>
__device__ __forceinline__ uint32_t chain_addr(uint32_t local, int rank) {
  if constexpr (CS == 1) return local;
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
  return r;
}
template <int CS>
__device__ __forceinline__ void chain_store(uint32_t addr, double v) {
  if constexpr (CS == 1)
    asm volatile("st.shared.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
  else
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
}

template <int L, int CS, int QS>
__global__ void __launch_bounds__(32 * ((1 << L) / CS), 8 / ((1 << L) / CS)) k_mc_chain(McArgs a) {
  constexpr int TW = 1 << L, W = TW / CS;
  static_assert(L >= 1 && L <= 6 && W >= 1 && W <= 8, "one chain per CTA or cluster");
  extern __shared__ __align__(128) unsigned char smraw[];
  double *buf = reinterpret_cast<double *>(smraw);         // W slices of 2048 values
  double *sums = buf + 2048 * W;                           // per warp of the chain: p2, m
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int rank = CS == 1 ? 0 : (int)(blockIdx.x % CS), c = blockIdx.x / CS;
  const int sw = rank * W + w;
  double *slice = buf + 2048 * w;
  uint32_t peer[CS];
#pragma unroll
  for (int k = 0; k < CS; ++k) peer[k] = chain_addr<CS>((uint32_t)__cvta_generic_to_shared(buf), k);
  McChain ch;
  ch.start(a, c);
  if constexpr (CS > 1) chain_sync<CS>();  // every CTA of the cluster runs before remote stores
  for (int t = 0; t < a.nsamples; ++t) {
    ch.fetch(a, t);
    double p2 = 0.0, m = 0.0;
    if (ch.prop != 0) {  // the same for all warps of the chain
      double2 v[32];
      wide_build(v, a.psi, (uint32_t)ch.prop, (uint32_t)(1024 * sw + lane), 0u);
      // put: register i of this warp holds bits 5 .. 9 = i
#pragma unroll
      for (int cl = 0; cl < 4; ++cl) {
        wht_class<2, 5>(v, cl);
#pragma unroll
        for (int i = cl; i < 32; i += 4) {
          const int lo = i & ((1 << (6 - L)) - 1), dw = i >> (6 - L);
          const uint32_t rl = (uint32_t)((lo << (L - 1)) | (sw >> 1));  // reading lane
          const uint32_t pos = ((uint32_t)sw << (11 - L) | (uint32_t)(lo << 5) | (uint32_t)lane) ^ ((rl & 7u) << 1);
          const int dr = dw, di = dw + TW / 2;  // warps of the real and the imaginary plane
          chain_store<CS>(peer[dr / W] + (uint32_t)((dr % W) * 2048) * 8u + pos * 8u, v[i].x);
          chain_store<CS>(peer[di / W] + (uint32_t)((di % W) * 2048) * 8u + pos * 8u, v[i].y);
        }
      }
      chain_sync<CS>();
      const uint32_t lo = (uint32_t)lane >> (L - 1), hi = (uint32_t)lane & ((1u << (L - 1)) - 1u);
#pragma unroll
      for (int b = 0; b < 2; ++b)
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const uint32_t pos = ((hi << 1 | b) << (11 - L) | lo << 5 | (uint32_t)(2 * i)) ^ (((uint32_t)lane & 7u) << 1);
          v[16 * b + i] = *reinterpret_cast<const double2 *>(slice + pos);
        }
      __syncwarp();
      double s[5];
      if constexpr (L <= 2) {
        if constexpr (L == 2) lane_wht(v, lane, 1);
        wide_moments<QS, 5, true>(v, s, a.qp, slice, lane);
      } else {
#pragma unroll
        for (int b = 0; b < 8; ++b) wht_block<0, 2>(v, b);
#pragma unroll
        for (int cl = 0; cl < 4; ++cl) wht_class<2, 5>(v, cl);
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const double p = v[i].x, q = v[i].y;
          v[i].x = p + q;
          v[i].y = p - q;
        }
        transpose_ab<32>(v, reinterpret_cast<double2 *>(slice), lane);
        wide_moments<QS, L - 1, false>(v, s, a.qp, slice, lane);
      }
      p2 = warp_sum(s[0]) * 4.0;
      m = warp_sum(s[1]) * moment_scale<QS>(a.qp);
      if (lane < CS) {
        const uint32_t dst = chain_addr<CS>((uint32_t)__cvta_generic_to_shared(sums + 2 * sw), lane);
        chain_store<CS>(dst, p2);
        chain_store<CS>(dst + 8u, m);
      }
      chain_sync<CS>();
      // all warps' sums in warp order: lanes take warps l and l + 32, then a fixed butterfly
      dd sp{0.0, 0.0}, sm{0.0, 0.0};
#pragma unroll
      for (int u = 0; u < (TW + 31) / 32; ++u)
        if (lane + 32 * u < TW) {
          dd_add(sp, sums[2 * (lane + 32 * u)]);
          dd_add(sm, sums[2 * (lane + 32 * u) + 1]);
        }
#pragma unroll
      for (int o = (TW < 32 ? TW : 32) / 2; o > 0; o >>= 1) {
        dd op, om;
        op.hi = __shfl_xor_sync(0xffffffffu, sp.hi, o);
        op.lo = __shfl_xor_sync(0xffffffffu, sp.lo, o);
        om.hi = __shfl_xor_sync(0xffffffffu, sm.hi, o);
        om.lo = __shfl_xor_sync(0xffffffffu, sm.lo, o);
        dd_add_dd(sp, op);
        dd_add_dd(sm, om);
      }
      p2 = __shfl_sync(0xffffffffu, sp.hi + sp.lo, 0);
      m = __shfl_sync(0xffffffffu, sm.hi + sm.lo, 0);
    }
    ch.step(a, p2, m);
  }
  if (sw == 0 && lane == 0) ch.finish(a, c);
}

// initial chain state: currPROB = 1e-120, currM2 = 0, currP2 = p2_0, first proposal
__global__ void k_mc_init(McArgs a) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c < a.nbeta) {
    Chain ch;
    ch.cur = 0;
    ch.prop = a.pd[(size_t)c * a.nsamples];
    ch.prob = 1e-120;
    ch.m2 = 0.0;
    ch.p2 = a.p2_0;
    ch.sM2 = ch.sM2sq = ch.sP2 = 0.0;
    ch.beta = (double)(a.chain0 + c) / (double)(a.nbeta_grid - 1);
    ch.n = 0;
    a.ch[c] = ch;
  }
  if (c == 0) {
    *a.step = 0;
    *a.upd_done = 0;
  }
}

// per-chain means and the Simpson combination -> out[0] = m2, out[1 + 3c ..] = (M2, M2ADD, P2)
__global__ void k_mc_finish(McArgs a, double *out, uint64_t *final_mask) {
  if (threadIdx.x != 0) return;
  const int nb = a.nbeta;
  const double h = 1.0 / (double)(nb - 1);
  double odd = 0.0, even = 0.0, odda = 0.0, evena = 0.0;
  const double m2add = a.m0 / (double)(1ull << a.n);
  for (int i = 0; i < nb; ++i) {
    const Chain ch = a.ch[i];
    const double M2 = ch.sM2 / (double)ch.n;
    out[1 + 3 * i] = M2;
    out[2 + 3 * i] = m2add;
    out[3 + 3 * i] = ch.sP2 / (double)ch.n;
    final_mask[i] = ch.cur;
    if (i > 0 && i < nb - 1) {
      if (i % 2 == 1) {
        odd += M2;
        odda += m2add;
      } else {
        even += M2;
        evena += m2add;
      }
    }
  }
  if (a.chain0 != 0 || nb != a.nbeta_grid) {
    out[0] = 0.0;  // a range of the grid: the caller combines all chains
    return;
  }
  const double M2_0 = out[1], M2_e = out[1 + 3 * (nb - 1)];
  const double I_res = (h / 3.0) * (M2_0 + M2_e + 4.0 * odd + 2.0 * even);
  const double I_add = (h / 3.0) * (m2add + m2add + 4.0 * odda + 2.0 * evena);
  out[0] = -log2(pow(2.0, -I_res) + I_add);
}

// One launch of a step kernel.  The kernels of consecutive steps are chained by
// programmatic dependent launch (the next grid is set up while this one runs); every kernel
// waits for its predecessor at its start, before any access to global memory, so the
// order of their effects is the plain stream order.  The first launch of a captured block
// is not chained: it waits for everything before it.
template <typename... P, typename... A>
static cudaError_t mc_launch(hm_ctx *c, bool chained, void (*kern)(P...), int blocks, int threads, size_t smem,
                             A &&...args) {
  cudaLaunchConfig_t lc = {};
  lc.gridDim = dim3(blocks);
  lc.blockDim = dim3(threads);
  lc.dynamicSmemBytes = smem;
  lc.stream = c->stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  lc.attrs = at;
  lc.numAttrs = chained ? 1 : 0;
  return cudaLaunchKernelEx(&lc, kern, std::forward<A>(args)...);
}

template <int QS>
int mc_enqueue_step(hm_ctx *c, McArgs &a, bool first) {
  const int n = a.n;
  const int upd_blocks = (a.nbeta + MC_UPD_WARPS - 1) / MC_UPD_WARPS;
  const int hi = n - 11;
  const size_t smem = 4 * 32 * 32 * sizeof(double2);
  const long long units = (long long)a.nbeta * a.U;
  const int blocks = (int)((units + 3) / 4);
#define HM_MCP(HIv)                                                                                     \
  case HIv:                                                                                             \
  HM_CUDA(c, cudaFuncSetAttribute(k_mc_p1<HIv>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)); \
  HM_CUDA(c, cudaFuncSetAttribute(k_mc_p2<HIv, QS>, cudaFuncAttributeMaxDynamicSharedMemorySize,         \
                                  (int)smem));                                                           \
  HM_CUDA(c, mc_launch(c, !first, k_mc_p1<HIv>, blocks, 128, smem, a));                               \
  HM_CUDA(c, mc_launch(c, true, k_mc_p2<HIv, QS>, blocks, 128, smem, a));                             \
  break;
  switch (hi) {
    HM_MCP(5)
    HM_MCP(6)
    HM_MCP(7)
    HM_MCP(8)
    HM_MCP(9)
    HM_MCP(10)
    default:
      return set_err(c, HM_ERR_SIZE, "MC: n = %d outside [16, 21]", n);
  }
#undef HM_MCP
  HM_CUDA(c, mc_launch(c, true, k_mc_update, upd_blocks, MC_UPD_WARPS * 32, 0, a));
  return HM_OK;
}

template <int L, int CS, int QS>
static int launch_chain(hm_ctx *c, const McArgs &a) {
  constexpr int TW = 1 << L, W = TW / CS;
  const size_t smem = (2048 * W + 2 * TW) * sizeof(double);
  auto kern = k_mc_chain<L, CS, QS>;
  HM_CUDA(c, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  cudaLaunchConfig_t lc = {};
  lc.gridDim = dim3(a.nbeta * CS);
  lc.blockDim = dim3(32 * W);
  lc.dynamicSmemBytes = smem;
  lc.stream = c->stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = CS;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  lc.attrs = at;
  lc.numAttrs = CS > 1 ? 1 : 0;
  HM_CUDA(c, cudaLaunchKernelEx(&lc, kern, a));
  return HM_OK;
}

// all steps of all chains in one launch
template <int QS>
static int launch_chains(hm_ctx *c, const McArgs &a) {
  switch (a.n) {
#define HM_MCW(N)                                                                                          \
  case N:                                                                                                  \
    HM_CUDA(c, cudaFuncSetAttribute(k_mc_chain_warp<N - 1, QS>, cudaFuncAttributeMaxDynamicSharedMemorySize, \
                                    (int)(1024 * sizeof(double2))));                                       \
    k_mc_chain_warp<N - 1, QS><<<a.nbeta, 32, 1024 * sizeof(double2), c->stream>>>(a);                      \
    HM_CUDA(c, cudaGetLastError());                                                                        \
    return HM_OK;
    HM_MCW(1)
    HM_MCW(2)
    HM_MCW(3)
    HM_MCW(4)
    HM_MCW(5)
    HM_MCW(6)
    HM_MCW(7)
    HM_MCW(8)
    HM_MCW(9)
    HM_MCW(10)
    HM_MCW(11)
#undef HM_MCW
    case 12: return launch_chain<1, 1, QS>(c, a);
    case 13: return launch_chain<2, 1, QS>(c, a);
    // as many CTAs to a chain as shorten a step while every chain still gets its own SMs:
    // n = 14 5.4 us per step with two, 6.2 with one (81 chains: 7.0 and 6.2); n = 15 5.7 with
    // eight, 6.0 with four, 7.8 with two; n = 16 6.9 with eight, 8.8 with four
    case 14:
      return 2 * a.nbeta <= c->num_sms ? launch_chain<3, 2, QS>(c, a) : launch_chain<3, 1, QS>(c, a);
    case 15:
      return 8 * a.nbeta <= c->num_sms ? launch_chain<4, 8, QS>(c, a) : launch_chain<4, 4, QS>(c, a);
    case 16: return launch_chain<5, 8, QS>(c, a);
    case 17: return launch_chain<6, 8, QS>(c, a);
    default: return set_err(c, HM_ERR_SIZE, "MC chains: n = %d outside [1, 17]", a.n);
  }
}

}  // namespace

// per-chain means and the combination, read back to the host
static int mc_results(hm_ctx *c, const McArgs &a, double *d_res, uint64_t *d_mask, double *out, uint64_t *final_mask) {
  HM_CUDA(c, cudaEventRecord(c->ev1, c->stream));
  k_mc_finish<<<1, 32, 0, c->stream>>>(a, d_res, d_mask);
  c->launches += 1;
  HM_CUDA(c, cudaGetLastError());
  HM_CUDA(c, cudaMemcpyAsync(out, d_res, (1 + 3 * a.nbeta) * sizeof(double), cudaMemcpyDeviceToHost, c->stream));
  if (final_mask)
    HM_CUDA(c, cudaMemcpyAsync(final_mask, d_mask, a.nbeta * sizeof(uint64_t), cudaMemcpyDeviceToHost, c->stream));
  HM_CUDA(c, cudaStreamSynchronize(c->stream));
  float ms = 0.f;
  HM_CUDA(c, cudaEventElapsedTime(&ms, c->ev0, c->ev1));
  c->last_ms = ms;
  return HM_OK;
}

int run_mc(hm_ctx *c, const double2 *psi, int n, double q, int nbeta_grid, int chain0, int nbeta, int nsamples,
           const uint64_t *pd_dev, const double *rs_dev, double p2_0, double m0, double *out /* 1 + 3 nbeta */,
           uint64_t *final_mask) {
  McArgs a;
  memset(&a, 0, sizeof a);
  a.psi = psi;
  a.n = n;
  a.nbeta = nbeta;
  a.chain0 = chain0;
  a.nbeta_grid = nbeta_grid;
  a.nsamples = nsamples;
  a.pd = pd_dev;
  a.rs = rs_dev;
  set_qparams(a.qp, &q, 1);
  const bool q2 = (q == 2.0);
  a.p2_0 = p2_0;
  a.m0 = m0;
  // device state: chains, step counter, per-tile partials, ring, relabelled copies
  const size_t len = (size_t)1 << n;
  // One launch per run: us per step at 13 / 81 chains, against three (two, n <= 11) launches
  // per step: n = 8 1.69 against 6.28, n = 11 2.5 / 2.6 against 7.1 / 9.4, n = 12 2.7 / 2.7
  // against 12.1 / 15.1, n = 14 5.3 / 6.2 against 12.1 / 17.2, n = 15 5.7 / 15.5 against
  // 12.6 / 20.7 (601 chains: 71 against 90).  At n = 16 and 17 a chain's cluster takes eight
  // SMs and its exchange crosses them (17 bytes per clock and SM), so that with many chains
  // the passes through L2 catch up: n = 16 6.9 against 13.0 at 13 chains, 17.0 against 18.5
  // at 41, 18.6 against 21.4 at 61, 26.7 each at 81.  At n = 17 sixteen clusters are resident
  // at a time: 10.2 against 17.2 at 15 chains, 19.4 against 17.0 at 17, 20.0 against 19.3 at 21.
  // The rule looks at the whole grid, so that a range of its chains takes the same route.
  const bool one_launch = n <= 15 || (n == 16 && nbeta_grid <= 64) || (n == 17 && nbeta_grid <= 16);
  if (!one_launch) {
    a.U = 1 << (n - 11);
    HM_TRY(ensure_dev(c, &c->d_inter, &c->inter_cap, (size_t)nbeta * (len / 2) * sizeof(double2)));
    a.inter = (double2 *)c->d_inter;
    HM_TRY(ensure_dev(c, &c->d_aux2, &c->aux2_cap, 10 * len * sizeof(double2)));
    k_psi_swapped<double2><<<c->num_sms * 8, 256, 0, c->stream>>>(psi, (double2 *)c->d_aux2, n, 10);
    c->launches += 1;
    for (int j = 0; j < 10; ++j) a.psi_sw[j] = (const double2 *)c->d_aux2 + (size_t)j * len;
  }
  const size_t part_bytes = (size_t)nbeta * (a.U > 0 ? a.U : 1) * 2 * sizeof(double);
  const size_t state_bytes = 256 + nbeta * sizeof(Chain) + part_bytes + (1 + 3 * nbeta) * sizeof(double) +
                             nbeta * sizeof(uint64_t) + 256;
  HM_TRY(ensure_dev(c, (void **)&c->d_out, &c->out_cap, state_bytes));
  char *base = (char *)c->d_out;
  a.step = (long long *)base;
  a.upd_done = (unsigned *)(base + 64);
  a.ch = (Chain *)(base + 256);
  a.part = (double *)(base + 256 + nbeta * sizeof(Chain));
  double *d_res = (double *)(base + 256 + nbeta * sizeof(Chain) + part_bytes);
  uint64_t *d_mask = (uint64_t *)(d_res + 1 + 3 * nbeta);
  if (one_launch) {
    HM_CUDA(c, cudaEventRecord(c->ev0, c->stream));
    HM_TRY(q2 ? launch_chains<QS_Q2>(c, a) : launch_chains<QS_GEN>(c, a));
    c->launches += 1;
    return mc_results(c, a, d_res, d_mask, out, final_mask);
  }
  k_mc_init<<<(nbeta + 127) / 128, 128, 0, c->stream>>>(a);
  c->launches += 1;
  HM_CUDA(c, cudaGetLastError());
  // capture a block of steps once, replay it
  const int G = 16;
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  HM_CUDA(c, cudaStreamSynchronize(c->stream));
  HM_CUDA(c, cudaEventRecord(c->ev0, c->stream));
  HM_CUDA(c, cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeThreadLocal));
  int rc = HM_OK;
  for (int s = 0; s < G && rc == HM_OK; ++s)
    rc = q2 ? mc_enqueue_step<QS_Q2>(c, a, s == 0) : mc_enqueue_step<QS_GEN>(c, a, s == 0);
  cudaError_t ce = cudaStreamEndCapture(c->stream, &graph);
  if (rc != HM_OK) {
    if (graph) cudaGraphDestroy(graph);
    return rc;
  }
  if (ce != cudaSuccess) return set_err(c, HM_ERR_CUDA, "MC graph capture failed: %s", cudaGetErrorString(ce));
  ce = cudaGraphInstantiate(&exec, graph, 0);
  cudaGraphDestroy(graph);
  if (ce != cudaSuccess) return set_err(c, HM_ERR_CUDA, "MC graph instantiation failed: %s", cudaGetErrorString(ce));
  for (int s = 0; s < nsamples; s += G) {
    ce = cudaGraphLaunch(exec, c->stream);
    if (ce != cudaSuccess) break;
    c->launches += G * 3;  // per step: the two passes and the update
  }
  cudaGraphExecDestroy(exec);
  if (ce != cudaSuccess) return set_err(c, HM_ERR_CUDA, "MC graph launch failed: %s", cudaGetErrorString(ce));
  return mc_results(c, a, d_res, d_mask, out, final_mask);
}

}  // namespace hm

namespace hm {
namespace {

// chains [cb, ce) of an nbeta-point grid; out: 1 + 3 (ce - cb) doubles
int mc_chains(hm_ctx *c, const double *psi, int n, double q, int nbeta, int cb, int ce, int nsamples,
              const uint64_t *prop_delta, const double *rs, double *out, uint64_t *final_mask) {
  if (!psi || !prop_delta || !rs) return set_err(c, HM_ERR_ARG, "null pointer");
  if (n < 1 || n > 21) return set_err(c, HM_ERR_SIZE, "MC: n = %d outside [1, 21]", n);
  if (nbeta < 3 || nbeta % 2 != 1 || nbeta > HM_MC_MAX_NBETA)
    return set_err(c, HM_ERR_ARG, "Simpson needs an odd number of beta points in [3, %d] (got %d)", HM_MC_MAX_NBETA,
                   nbeta);
  if (cb < 0 || ce > nbeta || cb >= ce)
    return set_err(c, HM_ERR_ARG, "chain range [%d, %d) outside the %d-point beta grid", cb, ce, nbeta);
  if (nsamples < 1) return set_err(c, HM_ERR_ARG, "nsamples must be >= 1");
  if (!(q >= 1.0 && q <= 16.0)) return set_err(c, HM_ERR_Q, "Renyi index q = %g outside [1, 16]", q);
  HM_CUDA(c, cudaSetDevice(c->device));
  c->launches = 0;
  const int nch = ce - cb;
  const size_t len = (size_t)1 << n;
  const size_t ns = (size_t)nch * nsamples;
  HM_TRY(ensure_dev(c, &c->d_psi, &c->psi_cap, len * sizeof(double2)));
  HM_CUDA(c, cudaMemcpyAsync(c->d_psi, psi, len * sizeof(double2), cudaMemcpyHostToDevice, c->stream));
  // m0 and p2_0 of x = 0 (sample_mask!(0), src/SRE.jl:147): one X-string of the exact
  // sweep, before the chains take the context's scratch buffers
  QReq qq;
  qq.nq = 1;
  qq.q[0] = q;
  double z[4];
  HM_TRY(run_sre(c, (const double2 *)c->d_psi, n, 0, 1, qq, HM_FP64, z));
  const double p2_0 = (z[0] + z[1]) / (double)len, m0 = z[2] + z[3];
  HM_TRY(ensure_dev(c, &c->d_aux, &c->aux_cap, ns * (sizeof(uint64_t) + sizeof(double))));
  uint64_t *pd = (uint64_t *)c->d_aux;
  double *r = (double *)(pd + ns);
  HM_CUDA(c, cudaMemcpyAsync(pd, prop_delta, ns * sizeof(uint64_t), cudaMemcpyHostToDevice, c->stream));
  HM_CUDA(c, cudaMemcpyAsync(r, rs, ns * sizeof(double), cudaMemcpyHostToDevice, c->stream));
  return run_mc(c, (const double2 *)c->d_psi, n, q, nbeta, cb, nch, nsamples, pd, r, p2_0, m0, out, final_mask);
}

}  // namespace
}  // namespace hm

extern "C" int hm_mc_sre(hm_ctx *c, const double *psi, int n, double q, int nbeta, int nsamples,
                         const uint64_t *prop_delta, const double *rs, double *out_m2, double *M2, double *M2ADD,
                         double *P2, uint64_t *final_mask) {
  if (!c) return HM_ERR_ARG;
  c->err.clear();
  if (!out_m2 || !M2 || !M2ADD || !P2) return hm::set_err(c, HM_ERR_ARG, "null pointer");
  if (nbeta < 3 || nbeta > HM_MC_MAX_NBETA)
    return hm::set_err(c, HM_ERR_ARG, "Simpson needs an odd number of beta points in [3, %d] (got %d)",
                       HM_MC_MAX_NBETA, nbeta);
  std::vector<double> out(1 + 3 * (size_t)nbeta);
  HM_TRY(hm::mc_chains(c, psi, n, q, nbeta, 0, nbeta, nsamples, prop_delta, rs, out.data(), final_mask));
  *out_m2 = out[0];
  for (int i = 0; i < nbeta; ++i) {
    M2[i] = out[1 + 3 * i];
    M2ADD[i] = out[2 + 3 * i];
    P2[i] = out[3 + 3 * i];
  }
  return HM_OK;
}

extern "C" int hm_mc_sre_chains(hm_ctx *c, const double *psi, int n, double q, int nbeta, int chain_begin,
                                int chain_end, int nsamples, const uint64_t *prop_delta, const double *rs, double *M2,
                                double *M2ADD, double *P2, uint64_t *final_mask) {
  if (!c) return HM_ERR_ARG;
  c->err.clear();
  if (!M2 || !M2ADD || !P2) return hm::set_err(c, HM_ERR_ARG, "null pointer");
  if (chain_begin < 0 || chain_end > nbeta || chain_begin >= chain_end || nbeta > HM_MC_MAX_NBETA)
    return hm::set_err(c, HM_ERR_ARG, "chain range [%d, %d) outside the %d-point beta grid", chain_begin, chain_end,
                       nbeta);
  std::vector<double> out(1 + 3 * (size_t)(chain_end - chain_begin));
  HM_TRY(hm::mc_chains(c, psi, n, q, nbeta, chain_begin, chain_end, nsamples, prop_delta, rs, out.data(),
                       final_mask));
  for (int i = 0; i < chain_end - chain_begin; ++i) {
    M2[i] = out[1 + 3 * i];
    M2ADD[i] = out[2 + 3 * i];
    P2[i] = out[3 + 3 * i];
  }
  return HM_OK;
}
