// sre_launch.cuh -- host launchers for the exact-SRE kernels (instantiated per precision and
// moment set in sre_fp64_q2.cu, sre_fp64_q23.cu, ...).
#pragma once
#include "hm_ctx.h"
#include "sre_kernels.cuh"
#include "sre_wide.cuh"
#include "sweep3.cuh"

namespace hm {

// The largest n whose X-strings one CTA holds (k_sre_wide); two passes from there up.
constexpr int single_cta_max(bool fp64) { return fp64 ? 14 : 15; }

// Two-pass sweeps that stay on k_sre_stage, FP64 (us per X-string on B200; the other side is
// k_sre_wide_stage at its best batch): n = 20, q = 2 X = 10 3.74 (X = 7 3.87), q = 2 and 3 3.85
// (q = 3 4.06); n = 19, q = 2 and 3 X = 16 1.84 (X = 9 1.89).  Both kernels are bound by the
// ring's traffic there, and its tensor stores need no group of four.
template <typename T, int QS> constexpr bool on_stage_kernel(int n) {
  return sizeof(T) == 8 && ((n == 20 && QS != QS_GEN) || (n == 19 && QS == QS_Q23));
}

// Tunables of the two-pass stage kernels (set through hm_set_param): a batch holds about
// `units_target` warp units per pass (X = units_target / 2^(n-11) X-strings, or X when set
// explicitly), the two-batch ring stays within `ring_mib`, and `graph_stages` stages are
// captured per CUDA graph.  A stage costs about 1.4 us beyond its rounds of items over the
// groups of warps, and a last round that is not full costs a whole one; the ring's size
// costs DRAM traffic once it outgrows the 126 MB L2.  The default batch `measured_x` is the
// best of those that give whole rounds (2 X 2^HI items over 592 groups of two warps:
// X = 37 m at n = 17) within a ring of about 120 MiB, timed on B200 (us per X-string):
//   FP64  n = 15: X = 148 (0.107; 74: 0.120)    n = 16: X = 111 (0.191; 74: 0.195, 37: 0.22)
//         n = 17: X = 55 (0.377; 37: 0.387)     n = 18: X = 27 (0.784; 18: 0.785, 37: 0.796)
//         n = 19: X = 9 (1.735; 14: 1.759, 4: 1.83)  n = 21: X = 4 (9.10; 3: 9.29, 2: 9.87)
//         n = 20, q other than 2, 3: X = 9 (q = 4 4.46, q = 2.7 18.3; 7: 4.40, 21.7; 10: 4.60, 19.3)
//   FP32  n = 16: X = 148 (0.106; 74: 0.124)
//         n = 17: X = 110 (0.197; 74: 0.204)    n = 18: X = 55 (0.403; 37: 0.413)
//         n = 19: X = 18 (0.861; 28: 0.878)     n = 20: X = 9 (1.97; 7: 2.02)
//         n = 21: X = 4 (4.65; 2: 4.90)
// Against the rows and tiles of k_sre_stage, which ran every size before: FP64 0.116, 0.206,
// 0.430, 0.852, 1.815, 3.79, 10.33 for n = 15 .. 21, FP32 0.115, 0.221, 0.446, 0.967, 2.70,
// 10.02 for n = 16 .. 21.
// hm_autotune measures and records a batch for the machine at hand; setting
// HM_PARAM_BATCH, _UNITS or _RING switches to the generic rule.
inline int measured_x(bool fp64, int n, bool stage_kernel) {
  static const int f64[7] = {148, 111, 55, 27, 9, 9, 4}, f32[7] = {0, 148, 110, 55, 18, 9, 4};
  if (n < 15 || n > 21) return 0;
  if (stage_kernel) return n == 19 ? 16 : 10;
  return (fp64 ? f64 : f32)[n - 15];
}

struct TwoPassCfg {
  int X = 0;
  int X_set = 0;
  int units_target = 4096;
  int ring_mib = 64;
  int graph_stages = 128;  // stages per captured graph (128: 0.4 % faster than 32 at n = 20)
  int adj_x = 0;  // X-strings per batch of the adjoint stage kernels (0: the default rule)
  // batch sizes chosen by hm_autotune, per precision (0 FP64, 1 FP32) and qubit count;
  // 0 = not tuned.  Used when HM_PARAM_BATCH is not set (see tuned_batch).
  int tuned_x[2][32] = {};
};
// hm_autotune times q = 2: its batch is that of the kernel that runs q = 2 at this size, and
// not of one that other moment sets run there
template <typename T, int QS> inline int tuned_batch(const TwoPassCfg &cfg, int n) {
  return on_stage_kernel<T, QS>(n) == on_stage_kernel<T, QS_Q2>(n) ? cfg.tuned_x[sizeof(T) == 8 ? 0 : 1][n] : 0;
}

TwoPassCfg &twopass_cfg();

// Tensor map of the two-pass ring for the pass-1 tensor stores (see p1_unit_tma):
// scalar_bytes 8 (FP64) or 4 (FP32), C positions per tile row, U = 2^HI rows, T tiles,
// two_x = 2X (slot, X-string) pairs, x_stride_bytes = 2^(n-1) complex.  Returns false
// (and leaves the plain stores in use) when the geometry does not meet the unit's rules
// or the driver does not provide the encoder.
bool encode_ring_tmap(CUtensorMap *m, void *ring, int scalar_bytes, int C, int U, int T, int two_x,
                      uint64_t x_stride_bytes, const TmaGeom &g);

inline TmaGeom ring_tma_geom(int C, int T) {
  TmaGeom g;
  g.C = C;
  g.box0 = 2 * C <= 256 ? 2 * C : 256;
  g.nb0 = 2 * C / g.box0;
  g.box2 = g.nb0 > 1 ? 1 : (T < 256 ? T : 256);
  g.nb2 = T / g.box2;
  return g;
}

template <typename T, int R, int NB, int QS>
static int launch_fused(hm_ctx *c, const SreArgs &a0, int *nwarps_out) {
  using V = typename VT<T>::V;
  SreArgs a = a0;
  constexpr int PB = ilog2c(R) + 5;
  const size_t smem = (size_t)FUSED_WARPS * 32 * R * sizeof(V);
  auto kern = k_sre_fused<T, R, NB, QS>;
  int occ = 0;
  HM_TRY(kernel_occ(c, kern, FUSED_WARPS * 32, smem, &occ));
  const uint64_t XPW = 1ull << (PB - NB);
  const uint64_t ngroups = (a.k_end - a.k_begin + XPW - 1) / XPW;
  uint64_t blocks = (ngroups + FUSED_WARPS - 1) / FUSED_WARPS;
  const uint64_t maxb = (uint64_t)c->num_sms * occ;
  if (blocks > maxb) blocks = maxb;
  if (blocks < 1) blocks = 1;
  const int nwarps = (int)blocks * FUSED_WARPS;
  HM_TRY(ensure_dev(c, (void **)&c->d_partials, &c->partials_cap,
                    sizeof(double) * 2 * (QSet<QS>::NQ + 1) * (size_t)nwarps));
  a.partials = c->d_partials;
  kern<<<(unsigned)blocks, FUSED_WARPS * 32, smem, c->stream>>>(a);
  c->launches += 1;
  HM_CUDA(c, cudaGetLastError());
  *nwarps_out = 0;  // folded by the kernel
  return HM_OK;
}

// n = 12, 13, 14 (FP64 also 11, FP32 15): one CTA of G = 2^(n-11) warps per X-string (see k_sre_wide).  n = 14 is
// the last size whose planes (128 KB in FP64) and registers (8 warps of 255) fit an SM; the
// two-pass sweep was half as fast at each of the three sizes (figures in sre_wide.cuh).
template <typename T, int G, int QS>
static int launch_wide(hm_ctx *c, const SreArgs &a0, int *nwarps_out) {
  SreArgs a = a0;
  const size_t smem = (size_t)2048 * G * sizeof(T);
  auto kern = k_sre_wide<T, G, QS>;
  int occ = 0;
  HM_TRY(kernel_occ(c, kern, 32 * G, smem, &occ));
  const uint64_t blocks = std::min<uint64_t>(a.k_end - a.k_begin, (uint64_t)c->num_sms * occ);
  const int nwarps = (int)blocks * G;
  HM_TRY(ensure_dev(c, (void **)&c->d_partials, &c->partials_cap,
                    sizeof(double) * 2 * (QSet<QS>::NQ + 1) * (size_t)nwarps));
  a.partials = c->d_partials;
  kern<<<(unsigned)blocks, 32 * G, smem, c->stream>>>(a);
  c->launches += 1;
  HM_CUDA(c, cudaGetLastError());
  *nwarps_out = 0;  // folded by the kernel
  return HM_OK;
}

// Launch the nst chained stage kernels of a sweep (node s runs stage s).  Up to 2 G stages, two
// graphs' worth, go out as direct launches: a stage runs longer than its launch takes (about
// 2 us), while capturing and instantiating a graph holds back the first stage by about 3 us a
// node, and the last replay runs up to G - 1 stages without a batch (B200: n = 19, 36 stages
// 1206 -> 1037 us per call, 129 stages 2439 -> 1985 us of kernels).  Under a bound of 32
// stages, ranges that the larger batches of that time ran in 32 to 100 stages had become 5
// to 14 % slower at n = 18 and 19.  Longer sweeps
// replay a captured graph of G stages, with a one-thread kernel advancing the stage base in
// device memory after every replay.
template <typename Kern, typename Args>
static int run_stage_chain(hm_ctx *c, Kern kern, Args &a, int nst, int blocks, int threads, size_t smem, int G,
                           const char *what) {
  auto launch = [&](int s) {
    a.node = s;
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3(blocks);
    lc.blockDim = dim3(threads);
    lc.dynamicSmemBytes = smem;
    lc.stream = c->stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    lc.attrs = at;
    lc.numAttrs = s > 0 ? 1 : 0;  // the first stage waits for everything before it
    return cudaLaunchKernelEx(&lc, kern, a);
  };
  cudaError_t ce = cudaSuccess;
  if (nst <= 2 * G) {
    for (int s = 0; s < nst && ce == cudaSuccess; ++s) ce = launch(s);
    c->launches += nst;
    if (ce != cudaSuccess) return set_err(c, HM_ERR_CUDA, "%s launch failed: %s", what, cudaGetErrorString(ce));
    return HM_OK;
  }
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  HM_CUDA(c, cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeThreadLocal));
  for (int s = 0; s < G && ce == cudaSuccess; ++s) ce = launch(s);
  if (ce == cudaSuccess) {
    k_stage_advance<<<1, 1, 0, c->stream>>>(a.stage, (unsigned)G);
    ce = cudaGetLastError();
  }
  const cudaError_t ce_end = cudaStreamEndCapture(c->stream, &graph);
  if (ce == cudaSuccess) ce = ce_end;
  if (ce != cudaSuccess) {
    if (graph) cudaGraphDestroy(graph);
    cudaGetLastError();
    return set_err(c, HM_ERR_CUDA, "%s graph capture failed: %s", what, cudaGetErrorString(ce));
  }
  ce = cudaGraphInstantiate(&exec, graph, 0);
  cudaGraphDestroy(graph);
  if (ce != cudaSuccess) return set_err(c, HM_ERR_CUDA, "%s graph instantiation failed: %s", what, cudaGetErrorString(ce));
  for (int s = 0; s < nst && ce == cudaSuccess; s += G) {
    ce = cudaGraphLaunch(exec, c->stream);
    c->launches += G + 1;
  }
  cudaGraphExecDestroy(exec);
  if (ce != cudaSuccess) return set_err(c, HM_ERR_CUDA, "%s graph launch failed: %s", what, cudaGetErrorString(ce));
  return HM_OK;
}

// Stage-kernel two-pass sweep (see k_sre_stage): X-strings per batch sized so that a
// pass holds about `units_target` warp units, ring of two batches, stages replayed from
// a captured CUDA graph.
template <typename T, int R, int HI, int QS>
static int launch_stages(hm_ctx *c, const SreArgs &a0, int *nwarps_out) {
  using V = typename VT<T>::V;
  const TwoPassCfg cfg = twopass_cfg();
  constexpr int PB = ilog2c(R) + 5, NQ = QSet<QS>::NQ;
  StageArgs a;
  memset(&a, 0, sizeof a);
  a.psi = a0.psi;
  a.k_begin = a0.k_begin;
  a.k_end = a0.k_end;
  a.qp = a0.qp;
  a.n = a0.n;
  const uint64_t U = 1ull << HI;
  const uint64_t len = a.k_end - a.k_begin;
  const TwoPassCfg def;
  const bool generic = cfg.X_set || cfg.units_target != def.units_target || cfg.ring_mib != def.ring_mib;
  uint64_t X, ring_mib = (uint64_t)cfg.ring_mib;
  const int tuned = tuned_batch<T, QS>(cfg, a.n);
  const int measured = generic ? 0 : measured_x(sizeof(T) == 8, a.n, true);
  if (cfg.X_set) {
    X = (uint64_t)cfg.X;
  } else if (tuned > 0 || measured > 0) {
    X = (uint64_t)(tuned > 0 ? tuned : measured);
    ring_mib = std::max<uint64_t>(ring_mib, (2 * X * ((uint64_t)1 << (a.n - 1)) * sizeof(V) + (1 << 20) - 1) >> 20);
  } else {
    X = std::max<uint64_t>(1, (uint64_t)cfg.units_target / U);
  }
  // ring bytes 2 X 2^(n-1) sizeof(V) within the budget
  const uint64_t per_x = ((uint64_t)1 << (a.n - 1)) * sizeof(V);
  while (X > 1 && 2 * X * per_x > (ring_mib << 20)) X >>= 1;
  if (X > len) X = len;
  a.X = (int)X;
  a.nbatch = (int)((len + X - 1) / X);
  const size_t ring_bytes = 2 * (size_t)X * per_x;
  HM_TRY(ensure_dev(c, &c->d_inter, &c->inter_cap, ring_bytes));
  a.ring = c->d_inter;
  {
    constexpr int C = 1 << (PB - HI), NT = (1 << PB) / C;
    a.g = ring_tma_geom(C, NT);
    a.tma = encode_ring_tmap(&a.tmap, a.ring, (int)sizeof(T), C, 1 << HI, NT, 2 * (int)X, per_x, a.g) ? 1 : 0;
  }
  if (a.k_begin < (1ull << PB) && a.k_end > 1) {  // some 0 < x < 2^PB in the range
    const size_t slen = (size_t)1 << a.n;
    HM_TRY(ensure_dev(c, &c->d_aux2, &c->aux2_cap, (size_t)PB * slen * sizeof(V)));
    k_psi_swapped<V><<<c->num_sms * 8, 256, 0, c->stream>>>(reinterpret_cast<const V *>(a.psi),
                                                            reinterpret_cast<V *>(c->d_aux2), a.n, PB);
    c->launches += 1;
    HM_CUDA(c, cudaGetLastError());
    for (int j = 0; j < PB; ++j) a.psi_sw[j] = reinterpret_cast<const V *>(c->d_aux2) + (size_t)j * slen;
  }
  const size_t smem = (size_t)SRE_WARPS * 32 * R * sizeof(V);
  auto kern = k_sre_stage<T, R, HI, QS>;
  int occ = 0;
  HM_TRY(kernel_occ(c, kern, SRE_WARPS * 32, smem, &occ));
  long long units = 2 * (long long)X * (long long)U;
  int blocks = c->num_sms * occ;
  if ((long long)blocks * SRE_WARPS > units) blocks = (int)((units + SRE_WARPS - 1) / SRE_WARPS);
  const int nwarps = blocks * SRE_WARPS;
  HM_TRY(ensure_dev(c, (void **)&c->d_partials, &c->partials_cap, sizeof(double) * 2 * (NQ + 1) * (size_t)nwarps));
  HM_CUDA(c, cudaMemsetAsync(c->d_partials, 0, sizeof(double) * 2 * (NQ + 1) * (size_t)nwarps, c->stream));
  a.slots = c->d_partials;
  HM_TRY(ensure_dev(c, (void **)&c->d_ctrl, &c->ctrl_cap, 4 * sizeof(unsigned)));
  HM_CUDA(c, cudaMemsetAsync(c->d_ctrl, 0, 4 * sizeof(unsigned), c->stream));
  a.stage = c->d_ctrl;
  const int nst = a.nbatch + 1;
  HM_TRY(run_stage_chain(c, kern, a, nst, blocks, SRE_WARPS * 32, smem, cfg.graph_stages, "stage"));
  *nwarps_out = nwarps;
  return HM_OK;
}

// Warps per pass-1 group of the two-pass sweep at n qubits: two (rows of 2048 complex
// values), more from the size on where pass 2 would otherwise hold more than one row bit on
// lane bits and read less than 128 bytes per row and unit (FP32 at n = 19: 0.861 us per
// X-string with four, 0.966 with two).  Past n = 20 the units of a warp are paired to whole
// lines anyway; FP64 at n = 21: 9.10 with four and pairs, 9.40 with eight.
template <typename T> constexpr int wide_group(int n) {
  return n <= (sizeof(T) == 8 ? 19 : 18) ? 2 : n <= (sizeof(T) == 8 ? 21 : 20) ? 4 : 8;
}

// Two-pass sweep (see k_sre_wide_stage): ring of two batches, stages chained and replayed
// from a captured CUDA graph.
template <typename T, int N, int QS>
static int launch_wide_stages(hm_ctx *c, const SreArgs &a0, int *nwarps_out) {
  constexpr int G = wide_group<T>(N), HI = N - 11 - ilog2c(G), NQ = QSet<QS>::NQ, WARPS = WideCta<G>::WARPS;
  const TwoPassCfg cfg = twopass_cfg();
  WideArgs a;
  memset(&a, 0, sizeof a);
  a.psi = a0.psi;
  a.k_begin = a0.k_begin;
  a.k_end = a0.k_end;
  a.qp = a0.qp;
  const uint64_t len = a.k_end - a.k_begin, per_x = ((uint64_t)1 << N) * sizeof(T);
  const TwoPassCfg def;
  const bool generic = cfg.X_set || cfg.units_target != def.units_target || cfg.ring_mib != def.ring_mib;
  uint64_t X, ring_mib = (uint64_t)cfg.ring_mib;
  const int tuned = tuned_batch<T, QS>(cfg, N);
  const int measured = generic ? 0 : measured_x(sizeof(T) == 8, N, false);
  if (cfg.X_set) {
    X = (uint64_t)cfg.X;
  } else if (tuned > 0 || measured > 0) {
    X = (uint64_t)(tuned > 0 ? tuned : measured);
    ring_mib = std::max<uint64_t>(ring_mib, (2 * X * per_x + (1 << 20) - 1) >> 20);
  } else {
    X = std::max<uint64_t>(1, (uint64_t)cfg.units_target >> (N - 11));
  }
  while (X > 1 && 2 * X * per_x > (ring_mib << 20)) X >>= 1;
  if (X > len) X = len;
  a.X = (int)X;
  a.nbatch = (int)((len + X - 1) / X);
  HM_TRY(ensure_dev(c, &c->d_inter, &c->inter_cap, 2 * (size_t)X * per_x));
  a.ring = c->d_inter;
  const size_t smem = (size_t)WARPS * 2048 * sizeof(T);
  auto kern = k_sre_wide_stage<T, G, HI, QS>;
  int occ = 0;
  HM_TRY(kernel_occ(c, kern, WARPS * 32, smem, &occ));
  const long long items = 2 * (long long)X << HI;
  const int blocks = (int)std::min<long long>((long long)c->num_sms * occ, (items * G + WARPS - 1) / WARPS);
  const int nwarps = blocks * WARPS;
  HM_TRY(ensure_dev(c, (void **)&c->d_partials, &c->partials_cap, sizeof(double) * 2 * (NQ + 1) * (size_t)nwarps));
  HM_CUDA(c, cudaMemsetAsync(c->d_partials, 0, sizeof(double) * 2 * (NQ + 1) * (size_t)nwarps, c->stream));
  a.slots = c->d_partials;
  HM_TRY(ensure_dev(c, (void **)&c->d_ctrl, &c->ctrl_cap, 4 * sizeof(unsigned)));
  HM_CUDA(c, cudaMemsetAsync(c->d_ctrl, 0, 4 * sizeof(unsigned), c->stream));
  a.stage = c->d_ctrl;
  HM_TRY(run_stage_chain(c, kern, a, a.nbatch + 1, blocks, WARPS * 32, smem, cfg.graph_stages, "stage"));
  *nwarps_out = nwarps;
  return HM_OK;
}

// Three-pass sweep for n = 21 + K (K = 1 .. 3): batch X (HM_PARAM_BATCH, else about 4096
// units per pass: X = 2 at n = 22, 1 above), ring of three batches, graph replay of
// programmatically chained stages as launch_stages.
template <typename T, int R, int K, int QS>
static int launch_stages3(hm_ctx *c, const SreArgs &a0, int *nwarps_out) {
  using V = typename VT<T>::V;
  const TwoPassCfg cfg = twopass_cfg();
  constexpr int PB = ilog2c(R) + 5, NQ = QSet<QS>::NQ;
  Stage3Args a;
  memset(&a, 0, sizeof a);
  a.psi = a0.psi;
  a.k_begin = a0.k_begin;
  a.k_end = a0.k_end;
  a.qp = a0.qp;
  a.n = a0.n;
  const uint64_t U = 1ull << (a.n - 11);
  const uint64_t len = a.k_end - a.k_begin;
  uint64_t X = cfg.X_set ? (uint64_t)cfg.X : std::max<uint64_t>(1, 4096 / U);
  if (X > len) X = len;
  a.X = (int)X;
  a.nbatch = (int)((len + X - 1) / X);
  const uint64_t per_x = ((uint64_t)1 << (a.n - 1)) * sizeof(V);
  HM_TRY(ensure_dev(c, &c->d_inter, &c->inter_cap, 3 * (size_t)X * per_x));
  a.ring = c->d_inter;
  {
    // the ring as 3 X 2^K sub-vectors in the n = 21 layout: rows of C = 1 position,
    // 1024 rows, 1024 tiles
    a.g = ring_tma_geom(1, 1 << PB);
    a.tma = encode_ring_tmap(&a.tmap, a.ring, (int)sizeof(T), 1, 1 << PB, 1 << PB, (int)(3 * X) << K,
                             ((uint64_t)1 << 20) * sizeof(V), a.g)
                ? 1
                : 0;
  }
  if (a.k_begin < (1ull << PB) && a.k_end > 1) {  // some 0 < x < 2^PB in the range
    const size_t slen = (size_t)1 << a.n;
    HM_TRY(ensure_dev(c, &c->d_aux2, &c->aux2_cap, (size_t)PB * slen * sizeof(V)));
    k_psi_swapped<V><<<c->num_sms * 8, 256, 0, c->stream>>>(reinterpret_cast<const V *>(a.psi),
                                                            reinterpret_cast<V *>(c->d_aux2), a.n, PB);
    c->launches += 1;
    HM_CUDA(c, cudaGetLastError());
    for (int j = 0; j < PB; ++j) a.psi_sw[j] = reinterpret_cast<const V *>(c->d_aux2) + (size_t)j * slen;
  }
  const size_t smem = (size_t)SRE_WARPS * 32 * R * sizeof(V);
  auto kern = k_sre_stage3<T, R, K, QS>;
  int occ = 0;
  HM_TRY(kernel_occ(c, kern, SRE_WARPS * 32, smem, &occ));
  const long long units = (long long)X * (long long)U;
  int blocks = c->num_sms * occ;
  if ((long long)blocks * SRE_WARPS > units) blocks = (int)((units + SRE_WARPS - 1) / SRE_WARPS);
  const int nwarps = blocks * SRE_WARPS;
  HM_TRY(ensure_dev(c, (void **)&c->d_partials, &c->partials_cap, sizeof(double) * 2 * (NQ + 1) * (size_t)nwarps));
  HM_CUDA(c, cudaMemsetAsync(c->d_partials, 0, sizeof(double) * 2 * (NQ + 1) * (size_t)nwarps, c->stream));
  a.slots = c->d_partials;
  HM_TRY(ensure_dev(c, (void **)&c->d_ctrl, &c->ctrl_cap, 4 * sizeof(unsigned)));
  HM_CUDA(c, cudaMemsetAsync(c->d_ctrl, 0, 4 * sizeof(unsigned), c->stream));
  a.stage = c->d_ctrl;
  const int nst = a.nbatch + 2;
  HM_TRY(run_stage_chain(c, kern, a, nst, blocks, SRE_WARPS * 32, smem, cfg.graph_stages, "three-pass"));
  *nwarps_out = nwarps;
  return HM_OK;
}

// Complex registers per lane of k_sre_fused.  Up to n = 10 the 2^n X-strings do not fill the
// SMs' warps and a warp's serial chain is the kernel's time, so a warp takes as few of them
// as keeps bits 5 and up in registers (bits 3 and 4 go to lane bits).  At n = 11 a warp per
// X-string fills them: FP64 takes the single-CTA kernel with one warp, whose exchange is
// half as wide; FP32 keeps the 32 registers.  SRE call of q = 2, FP64 on B200, 32 registers
// everywhere -> this: n = 6 41.7 -> 37.8 us, 8 38.9 -> 34.0, 9 39.0 -> 36.7, 10 41.6 -> 40.0,
// 11 55.7 -> 47.3.
constexpr int fused_regs(int nb) { return nb <= 8 ? 8 : nb == 9 ? 16 : 32; }

#define HM_FUSED_CASE(NBv)                                         \
  case NBv:                                                        \
    return launch_fused<T, fused_regs(NBv), NBv, QS>(c, a, nw);
template <typename T, int R, int QS>
static int dispatch_sre(hm_ctx *c, const SreArgs &a, int *nw) {
  constexpr int PB = ilog2c(R) + 5;
  const int nb = a.n - 1;
  if (nb <= PB) {
    switch (nb) {
      HM_FUSED_CASE(0)
      HM_FUSED_CASE(1)
      HM_FUSED_CASE(2)
      HM_FUSED_CASE(3)
      HM_FUSED_CASE(4)
      HM_FUSED_CASE(5)
      HM_FUSED_CASE(6)
      HM_FUSED_CASE(7)
      HM_FUSED_CASE(8)
      HM_FUSED_CASE(9)
      case 10:
        if constexpr (sizeof(T) == 8)
          return launch_wide<T, 1, QS>(c, a, nw);
        else
          return launch_fused<T, 32, 10, QS>(c, a, nw);
      default:
        break;
    }
  } else {
    switch (nb - PB) {
      case 1:
        return launch_wide<T, 2, QS>(c, a, nw);
      case 2:
        return launch_wide<T, 4, QS>(c, a, nw);
      case 3:
        return launch_wide<T, 8, QS>(c, a, nw);
      case 4:
        if constexpr (sizeof(T) == 4)
          return launch_wide<T, 16, QS>(c, a, nw);
        else
          return launch_wide_stages<T, 15, QS>(c, a, nw);
      case 5:
        return launch_wide_stages<T, 16, QS>(c, a, nw);
      case 6:
        return launch_wide_stages<T, 17, QS>(c, a, nw);
      case 7:
        return launch_wide_stages<T, 18, QS>(c, a, nw);
      case 8:
        if constexpr (on_stage_kernel<T, QS>(19))
          return launch_stages<T, R, 8, QS>(c, a, nw);
        else
          return launch_wide_stages<T, 19, QS>(c, a, nw);
      case 9:
        if constexpr (on_stage_kernel<T, QS>(20))
          return launch_stages<T, R, 9, QS>(c, a, nw);
        else
          return launch_wide_stages<T, 20, QS>(c, a, nw);
      case 10:
        return launch_wide_stages<T, 21, QS>(c, a, nw);
      case 11:
        if constexpr (R == 32) return launch_stages3<T, R, 1, QS>(c, a, nw);
        break;
      case 12:
        if constexpr (R == 32) return launch_stages3<T, R, 2, QS>(c, a, nw);
        break;
      case 13:
        if constexpr (R == 32) return launch_stages3<T, R, 3, QS>(c, a, nw);
        break;
      default:
        break;
    }
  }
  return set_err(c, HM_ERR_SIZE, "n = %d outside the fused range of this precision", a.n);
}

// One precision and moment set.  nwarps = 0: the kernel wrote the folded sums to `out`;
// otherwise the number of per-warp partial records left to fold.
template <typename T, int R, int QS>
int launch_sre_qs(hm_ctx *c, const void *psi_dev, int n, uint64_t kb, uint64_t ke, const QParams &qp,
                  double *out, int *nwarps) {
  SreArgs a;
  memset(&a, 0, sizeof a);
  a.out = out;
  a.ticket = c->d_ticket;
  a.psi = psi_dev;
  a.n = n;
  a.k_begin = kb;
  a.k_end = ke;
  a.qp = qp;
  return dispatch_sre<T, R, QS>(c, a, nwarps);
}

// one translation unit per precision and moment set holds the kernels (sre_fp64_q2.cu, ...)
#define HM_EXTERN_SRE(T, QS)                                                                             \
  extern template int launch_sre_qs<T, 32, QS>(hm_ctx *, const void *, int, uint64_t, uint64_t,          \
                                               const QParams &, double *, int *);
HM_EXTERN_SRE(double, QS_Q2)
HM_EXTERN_SRE(double, QS_Q23)
HM_EXTERN_SRE(double, QS_GEN)
HM_EXTERN_SRE(float, QS_Q2)
HM_EXTERN_SRE(float, QS_Q23)
HM_EXTERN_SRE(float, QS_GEN)
#undef HM_EXTERN_SRE

}  // namespace hm
