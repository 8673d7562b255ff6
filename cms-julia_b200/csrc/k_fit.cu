// Broken-line fits of the chain's tuples (launchBrokenLineKernelsOnCPU,
// broken_line_fit_on_gpu.jl:166-203: 3-hit and 4-hit tuples, 5-hit tuples fitted
// with their first 4 hits, at most 24576 per multiplicity) and the stand-alone
// fit entry point pxl_bl_fit (3..8 hits, FP64 or mixed precision).
#include <algorithm>
#include <cstddef>

#include "../../include/pxl.h"
#include "bl_fit.cuh"
#include "pxl_internal.cuh"

namespace pxl {

namespace {

// Mixed precision keeps q/pT within 1e-5 of FP64 up to pT of about 100 GeV; the few stiffer
// tuples (about 1 % of a PU50 event's tuples are above 50 GeV) are fitted again in FP64.
constexpr double kRefitPt = 50.0;

// Returns false, writing nothing, for a mixed-precision fit that needs the FP64 refit.
template <int N, class T>
__device__ bool fit_tuple(const Dev& d, uint64_t g, uint32_t hb, const uint32_t* hits_of_tuple, double B) {
  double h[3][N];
  float ge[6][N];
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const uint32_t hit = hb + hits_of_tuple[i];
    const int det = d.detind[hit];
    const DetParamsD& dp = d.c.det[det];
    float gl[6];
    bl::to_global_cov(dp.R, d.xerr[hit], 0.0f, d.yerr[hit], gl);
#pragma unroll
    for (int k = 0; k < 6; ++k) ge[k][i] = gl[k];
    h[0][i] = d.xg[hit];
    h[1][i] = d.yg[hit];
    h[2][i] = d.zg[hit];
  }
  bl::TrackOut o;
  const bool ok = bl::fit_track<N, T>(h, ge, B, o);
  if (sizeof(T) == 4 && !(o.pt < kRefitPt)) return false;
  float* st = d.t_state + 5 * g;
  float* cv = d.t_cov + 15 * g;
#pragma unroll
  for (int k = 0; k < 5; ++k) st[k] = float(o.state[k]);
#pragma unroll
  for (int k = 0; k < 15; ++k) cv[k] = float(o.cov[k]);
  d.t_pt[g] = float(o.pt);
  d.t_eta[g] = float(o.eta);
  d.t_chi2[g] = float((o.chi2_line + o.chi2_circle) / double(2 * N - 5));
  d.t_fitted[g] = 1;
  (void)ok;
  return true;
}

// Which tuples are fitted, and with how many hits: 3-hit tuples with 3, 4- and
// 5-hit tuples with 4 (fit5as4), none flagged duplicate, at most fits_per_mult
// per multiplicity (the bin is read in decreasing id, so the largest ids win).
// The fitted tuples go to the event's region of fit_list (3-hit from the front, 4-hit from the
// back) so that every warp of the fit kernel runs one hit count; the others get zero outputs here.
// A block takes 256 tuples at a time: their list slots with one atomic per hit count, then the
// state and covariance words of the tuples left out, in word order so that the stores coalesce. An
// event has blocks as event_blocks gives them (one block took 580 us for the 51 k tuples of an event
// of pileup 170); its counters are cleared before the launch.
__global__ void __launch_bounds__(256) k_fit_list(Dev d) {
  pdl_sync(d);
  const int e = blockIdx.y;
  EvInfo& E = d.ev[e];
  __shared__ uint32_t s_n[2], s_base[2];
  __shared__ uint8_t s_fit[256];
  const uint64_t tb = E.tuple_base;
  const uint32_t nt = E.n_tuples;
  const unsigned lane = threadIdx.x & 31u, below = (1u << lane) - 1u;
  for (uint32_t t0 = blockIdx.x * 256u; t0 < nt; t0 += gridDim.x * 256u) {
    const uint32_t t = t0 + threadIdx.x;
    const uint64_t g = tb + t;
    if (threadIdx.x < 2) s_n[threadIdx.x] = 0;
    __syncthreads();
    bool fit = false;
    uint32_t n = 0;
    if (t < nt) {
      n = d.tuple_off[g + 1] - d.tuple_off[g];
      fit = n >= 3 && n <= 5 && d.quality[g] != 1;
      if (fit) {
        const uint32_t cnt = E.tm_off[n] - E.tm_off[n - 1];
        if (cnt > d.fits_per_mult) {
          uint32_t larger = 0;
          for (uint32_t u = t + 1; u < nt; ++u) {
            const uint64_t gu = tb + u;
            if (d.tuple_off[gu + 1] - d.tuple_off[gu] == n && d.quality[gu] != 1) ++larger;
          }
          fit = larger < d.fits_per_mult;
        }
      }
      d.t_fitted[g] = fit ? 1 : 0;
      if (!fit) { d.t_pt[g] = 0.f; d.t_eta[g] = 0.f; d.t_chi2[g] = 0.f; }
    }
    s_fit[threadIdx.x] = fit ? 1 : 0;
    const unsigned m3 = __ballot_sync(0xffffffffu, fit && n == 3);
    const unsigned m4 = __ballot_sync(0xffffffffu, fit && n != 3);
    uint32_t w3 = 0, w4 = 0;
    if (lane == 0) {
      if (m3) w3 = atomicAdd(&s_n[0], uint32_t(__popc(m3)));
      if (m4) w4 = atomicAdd(&s_n[1], uint32_t(__popc(m4)));
    }
    w3 = __shfl_sync(0xffffffffu, w3, 0);
    w4 = __shfl_sync(0xffffffffu, w4, 0);
    __syncthreads();
    if (threadIdx.x < 2 && s_n[threadIdx.x]) s_base[threadIdx.x] = atomicAdd(threadIdx.x ? &E.n_fit4 : &E.n_fit3, s_n[threadIdx.x]);
    __syncthreads();
    if (fit) {
      if (n == 3) d.fit_list[tb + s_base[0] + w3 + __popc(m3 & below)] = t;
      else d.fit_list[tb + nt - 1 - (s_base[1] + w4 + __popc(m4 & below))] = t;
    }
    const uint32_t m = nt - t0 < 256u ? nt - t0 : 256u;
    for (uint32_t w = threadIdx.x; w < 5 * m; w += 256u)
      if (!s_fit[w / 5]) d.t_state[5 * (tb + t0) + w] = 0.f;
    for (uint32_t w = threadIdx.x; w < 15 * m; w += 256u)
      if (!s_fit[w / 15]) d.t_cov[15 * (tb + t0) + w] = 0.f;
    __syncthreads();
  }
}

// The event's fits of one hit count (N), listed in `list` as fit_list lists them.
template <int N, class T, bool kRefit>
__device__ __forceinline__ void fit_event(const Dev& d, int e) {
  const EvInfo& E = d.ev[e];
  const uint64_t tb = E.tuple_base;
  const uint32_t hb = E.hit_base;
  const uint32_t nt = E.n_tuples;
  const uint32_t nfit = kRefit ? (N == 3 ? E.n_refit3 : E.n_refit4) : (N == 3 ? E.n_fit3 : E.n_fit4);
  const uint32_t* list = kRefit ? d.refit_list : d.fit_list;
  // B = Float64(Float32(bf)) as HelixFitOnGPU stores the field (ca_hit_ntuplet_generator.jl:83)
  const double B = double(d.c.b_field);
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nfit; i += gridDim.x * blockDim.x) {
    const uint32_t t = list[N == 3 ? tb + i : tb + nt - 1 - i];
    const uint64_t g = tb + t;
    if (!fit_tuple<N, T>(d, g, hb, d.tuple_hits + d.tuple_off[g], B)) {
      EvInfo& Ew = d.ev[e];
      const uint32_t k = atomicAdd(N == 3 ? &Ew.n_refit3 : &Ew.n_refit4, 1u);
      d.refit_list[N == 3 ? tb + k : tb + nt - 1 - k] = t;
    }
  }
}

// Both hit counts in one launch (blockIdx.z), each block one of them: a small batch waits for the longer
// one only (29 us for the two of one event, 15 together). 128 registers (four blocks per SM): the 4-hit
// fit spills a few hundred bytes to L1 but runs twice the warps, which hides more of its FP64 latency.
// kRefit: the FP64 refits of the mixed-precision fits that asked for one.
template <class T, bool kRefit>
__global__ void __launch_bounds__(128, 4) k_fit_tuples(Dev d) {
  pdl_sync(d);
  if (blockIdx.z == 0) fit_event<4, T, kRefit>(d, blockIdx.y);
  else fit_event<3, T, kRefit>(d, blockIdx.y);
}

template <int N, class T>
__device__ void standalone_fit(const double* hits, const float* hits_ge, int32_t first, double B, float* state,
                               float* cov, float* chi2, float* pt, float* eta, int32_t* status, int32_t t) {
  double h[3][N];
  float ge[6][N];
#pragma unroll
  for (int i = 0; i < N; ++i) {
#pragma unroll
    for (int a = 0; a < 3; ++a) h[a][i] = hits[3 * (first + i) + a];
#pragma unroll
    for (int k = 0; k < 6; ++k) ge[k][i] = hits_ge[6 * (first + i) + k];
  }
  bl::TrackOut o;
  const bool ok = bl::fit_track<N, T>(h, ge, B, o);
#pragma unroll
  for (int k = 0; k < 5; ++k) state[5 * t + k] = float(o.state[k]);
#pragma unroll
  for (int k = 0; k < 15; ++k) cov[15 * t + k] = float(o.cov[k]);
  chi2[t] = float((o.chi2_line + o.chi2_circle) / double(2 * N - 5));
  pt[t] = float(o.pt);
  eta[t] = float(o.eta);
  status[t] = ok ? 0 : 1;
}

}  // namespace

// ------------------------------------------------------------ hit-count buckets
// Stand-alone fits take tracks of 3..8 hits in any order. The track indices go to one list per hit
// count in the caller's workspace, so that every warp of the fits runs one hit count. Workspace:
// FitPlan header, then the lists. A list keeps the tracks in runs of the input order (a block's
// tracks of one hit count, warp by warp): the fits' loads and stores of neighbouring tracks then
// share their lines, and a block takes one global atomic per hit count. One global atomic per track
// on the six cursors took 317 us for 2^20 tracks, a third of the whole mixed-precision call.
constexpr int kPlanThreads = 256;
constexpr int kPlanPerThread = 16;      // tracks per thread of the two-kernel form
constexpr int32_t kPlanOneCta = 8192;   // up to here one CTA builds the plan in one launch

// tracks of each hit count among the block's range [t0, t1), added to s_cnt; a track of another hit
// count gets status -1
__device__ __forceinline__ void plan_count(const int32_t* __restrict__ offs, int32_t t0, int32_t t1, int32_t* status,
                                           uint32_t* s_cnt) {
  const unsigned lane = threadIdx.x & 31u;
  for (int32_t b = t0; b < t1; b += int32_t(blockDim.x)) {
    const int32_t t = b + int32_t(threadIdx.x);
    const int32_t nh = t < t1 ? offs[t + 1] - offs[t] : 0;
    if (t < t1 && status && (nh < 3 || nh > kFitMaxN)) status[t] = -1;
#pragma unroll
    for (int n = 3; n <= kFitMaxN; ++n) {
      const uint32_t m = __ballot_sync(0xffffffffu, nh == n);
      if (lane == 0 && m) atomicAdd(&s_cnt[n], uint32_t(__popc(m)));
    }
  }
}

// list entries of the block's tracks from the positions s_cur on
__device__ __forceinline__ void plan_fill(const int32_t* __restrict__ offs, int32_t t0, int32_t t1, int32_t* list,
                                          uint32_t* s_cur) {
  const unsigned lane = threadIdx.x & 31u, lt = (1u << lane) - 1u;
  for (int32_t b = t0; b < t1; b += int32_t(blockDim.x)) {
    const int32_t t = b + int32_t(threadIdx.x);
    const int32_t nh = t < t1 ? offs[t + 1] - offs[t] : 0;
#pragma unroll
    for (int n = 3; n <= kFitMaxN; ++n) {
      const uint32_t m = __ballot_sync(0xffffffffu, nh == n);
      uint32_t at = 0;
      if (lane == 0 && m) at = atomicAdd(&s_cur[n], uint32_t(__popc(m)));
      at = __shfl_sync(0xffffffffu, at, 0);
      if (nh == n) list[at + __popc(m & lt)] = t;
    }
  }
}

__global__ void __launch_bounds__(kPlanThreads) k_fit_plan_count(const int32_t* __restrict__ offs, int32_t n, FitPlan* plan,
                                                                 int32_t* status) {
  __shared__ uint32_t s_cnt[kFitMaxN + 1];
  if (threadIdx.x <= kFitMaxN) s_cnt[threadIdx.x] = 0;
  __syncthreads();
  const int32_t t0 = blockIdx.x * (kPlanThreads * kPlanPerThread);
  plan_count(offs, t0, min(n, t0 + kPlanThreads * kPlanPerThread), status, s_cnt);
  __syncthreads();
  if (threadIdx.x <= kFitMaxN && s_cnt[threadIdx.x]) atomicAdd(&plan->count[threadIdx.x], s_cnt[threadIdx.x]);
}

__global__ void __launch_bounds__(kPlanThreads) k_fit_plan_fill(const int32_t* __restrict__ offs, int32_t n, FitPlan* plan) {
  __shared__ uint32_t s_cur[kFitMaxN + 1];
  if (threadIdx.x <= kFitMaxN) s_cur[threadIdx.x] = 0;
  __syncthreads();
  const int32_t t0 = blockIdx.x * (kPlanThreads * kPlanPerThread), t1 = min(n, t0 + kPlanThreads * kPlanPerThread);
  plan_count(offs, t0, t1, nullptr, s_cur);
  __syncthreads();
  if (threadIdx.x <= kFitMaxN) {
    uint32_t base = 0;
    for (int k = 3; k < int(threadIdx.x); ++k) base += plan->count[k];
    const uint32_t c = s_cur[threadIdx.x];
    s_cur[threadIdx.x] = base + (c ? atomicAdd(&plan->cursor[threadIdx.x], c) : 0u);
    if (blockIdx.x == 0) plan->base[threadIdx.x] = base;
  }
  __syncthreads();
  plan_fill(offs, t0, t1, plan->list, s_cur);
}

__global__ void __launch_bounds__(1024) k_fit_plan_one(const int32_t* __restrict__ offs, int32_t n, FitPlan* plan,
                                                       int32_t* status) {
  pdl_trigger();
  __shared__ uint32_t s_cnt[kFitMaxN + 1], s_cur[kFitMaxN + 1];
  if (threadIdx.x <= kFitMaxN) s_cnt[threadIdx.x] = 0;
  __syncthreads();
  plan_count(offs, 0, n, status, s_cnt);
  __syncthreads();
  if (threadIdx.x <= kFitMaxN) {
    uint32_t base = 0;
    for (int k = 3; k < int(threadIdx.x); ++k) base += s_cnt[k];
    s_cur[threadIdx.x] = base;
    plan->count[threadIdx.x] = s_cnt[threadIdx.x];
    plan->base[threadIdx.x] = base;
  }
  __syncthreads();
  plan_fill(offs, 0, n, plan->list, s_cur);
}

namespace {

// One launch for all hit counts, where six launches on three streams, forked and joined by events,
// left each kernel's tail and the event waits (1237 mixed fits 43 us, now 28; 99991 FP64 fits 98 us,
// now 81).
constexpr int kFitResident = 4;  // blocks per SM: 128 registers a thread

// A block per 128 tracks, long fits first, so that the blocks even out; from four waves on one wave
// of blocks that go on to further tracks saves the blocks' starts (2^20 mixed fits 374 us instead
// of 416 with contracted FP32 arithmetic; 408 us with f32, which rounds each operation), which at 1.3
// waves costs more in balance than it saves (99991 FP64 fits 92 us instead of 81).
inline int bl_fit_blocks(int32_t n) {
  const int all = fit_blocks(n), wave = 148 * kFitResident;
  return all < 4 * wave ? all : wave;
}

template <class T>
__global__ void __launch_bounds__(kFitThreads, kFitResident) k_fit_buckets(const double* __restrict__ hits, const float* __restrict__ ge,
                                                    const int32_t* __restrict__ offs, const FitPlan* __restrict__ plan,
                                                    double B, float* state, float* cov, float* chi2, float* pt,
                                                    float* eta, int32_t* status) {
  pdl_sync();
  for_bucket_track(*plan, [&](auto n, int32_t t) {
    standalone_fit<decltype(n)::value, T>(hits, ge, offs[t], B, state, cov, chi2, pt, eta, status, t);
  });
}

}  // namespace

static_assert(offsetof(EvInfo, n_refit4) == offsetof(EvInfo, n_fit3) + 3 * sizeof(uint32_t), "cleared together");

void launch_fit(const Dev& d, const Launch& L) {
  // the events' n_fit3, n_fit4, n_refit3, n_refit4
  cudaMemset2DAsync(&d.ev[0].n_fit3, sizeof(EvInfo), 0, 4 * sizeof(uint32_t), size_t(d.E), L.s);
  L.run(k_fit_list, dim3(event_blocks(d.E, 148 * 4, 64), d.E), 256, 0, d);
  L.mark("fit_list");
  // about 7000 fits per PU50 event: enough CTAs for every SM with few events
  const int bx = (L.tune && L.tune[kTuneFitTuples] > 0) ? L.tune[kTuneFitTuples]
                                                         : std::max(2, std::min(64, (148 * 16) / std::max(1, int(d.E))));
  // FP64 as the reference fits (broken_line_fit_on_gpu.jl:28-30), or the mixed-precision fit
  const dim3 grid(bx, d.E, 2);
  if (d.fit_precision == 1) {
    L.run(k_fit_tuples<bl::f32, false>, grid, 128, 0, d);
    L.mark("broken_line_fit");
    // about 1 % of the fits: one block per event and hit count, more where an event has the GPU
    // to itself (a block's fits follow one another)
    L.run(k_fit_tuples<double, true>, dim3(event_blocks(d.E, 148, 16), d.E, 2), 128, 0, d);
    L.mark("broken_line_refit_fp64");
  } else {
    L.run(k_fit_tuples<double, false>, grid, 128, 0, d);
    L.mark("broken_line_fit");
  }
}

int64_t fit_plan_bytes(int32_t n_tracks) {
  return (int64_t(sizeof(FitPlan)) + 4 * int64_t(n_tracks > 0 ? n_tracks : 0) + 255) / 256 * 256;
}

int fit_plan_build(const int32_t* offs, int32_t n, FitPlan* plan, int32_t* status, cudaStream_t s) {
  const Launch L{s};
  if (n <= kPlanOneCta) {
    // one launch instead of a clear, a count and a fill; above, one CTA takes longer than they do
    L.run(k_fit_plan_one, 1, 1024, 0, offs, n, plan, status);
  } else {
    if (cudaMemsetAsync(plan, 0, sizeof(FitPlan) - sizeof(plan->list), s) != cudaSuccess) return PXL_ERR_CUDA;
    const int blocks = div_up(n, kPlanThreads * kPlanPerThread);
    L.run(k_fit_plan_count, blocks, kPlanThreads, 0, offs, n, plan, status);
    L.run(k_fit_plan_fill, blocks, kPlanThreads, 0, offs, n, plan);
  }
  return cudaGetLastError() == cudaSuccess ? 0 : PXL_ERR_CUDA;
}

}  // namespace pxl

extern "C" int64_t pxl_fit_workspace_bytes(int32_t n_tracks) { return pxl::fit_plan_bytes(n_tracks); }

extern "C" int32_t pxl_bl_fit(const double* hits, const float* hits_ge, const int32_t* offs, int32_t n, double b_field,
                              int32_t precision, float* state, float* cov, float* chi2, float* pt, float* eta,
                              int32_t* status, void* workspace, int64_t workspace_bytes, void* stream) {
  if (n < 0 || !hits || !hits_ge || !offs || !state || !cov || !chi2 || !pt || !eta || !status || !workspace)
    return PXL_ERR_ARG;
  if (precision != 0 && precision != 1) return PXL_ERR_ARG;
  if (workspace_bytes < pxl::fit_plan_bytes(n)) return PXL_ERR_CAPACITY;
  if (n == 0) return 0;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  auto* plan = static_cast<pxl::FitPlan*>(workspace);
  int rc = pxl::fit_plan_build(offs, n, plan, status, s);
  if (rc) return rc;
  pxl::Launch L{s};
  L.pdl = true;
  const int g = pxl::bl_fit_blocks(n);
  if (precision == 0)
    L.run(pxl::k_fit_buckets<double>, g, pxl::kFitThreads, 0, hits, hits_ge, offs, plan, b_field, state, cov, chi2, pt, eta, status);
  else
    L.run(pxl::k_fit_buckets<pxl::bl::f32>, g, pxl::kFitThreads, 0, hits, hits_ge, offs, plan, b_field, state, cov, chi2, pt, eta, status);
  return cudaGetLastError() == cudaSuccess ? 0 : PXL_ERR_CUDA;
}
