// Cellular automaton: doublets, outer-hit lists, cell connection, fishbone,
// ntuplet search, cell -> track lists, early duplicate removal and tuple
// multiplicity. Restates gpu_pixel_doublets.jl:19-360 (doublets_from_histo),
// gpu_ca_cell.jl:130-270, gpu_fishbone.jl:4-63, circle_eq.jl:18-93 and
// ca_hit_ntuplet_generator_kernels_impl.jl:45-211.
//
// Output order equals the serial reference's: doublets are counted per work item
// (inner hit x layer pair), scanned and written in the reference's loop order (so
// doublet ids are the reference's ids); per-key lists (cells ending on a hit,
// neighbours of a cell, tracks of a cell) are filled with atomics at the offsets of a
// shifted scan and then sorted, which restores the reference's push order (ascending
// producer index); tuples are counted per start cell, scanned, and written in the
// reference's depth-first order, so tuple ids match too. The doublet and connection
// tests lay their (item, candidate) and (cell, candidate) pairs end to end over the
// lanes of a warp, so that lanes stay busy whatever the candidate counts; the tuple
// walks run from per-warp queues of the start cells that walk, one tree per lane.
#include <algorithm>
#include <cstddef>

#include "alignment.cuh"
#include "doublet_staging.cuh"
#include "pxl_internal.cuh"

namespace pxl {

namespace {

__constant__ uint8_t c_layer_pairs[2 * kNPairs] = {0, 1, 0, 4, 0, 7, 1, 2, 1, 4, 1, 7, 4, 5, 7, 8, 2, 3, 2, 4,
                                                   2, 7, 5, 6, 8, 9, 0, 2, 1, 3, 0, 5, 0, 8, 4, 6, 7, 9};
__constant__ int16_t c_phi_cuts[kNPairs] = {522, 730, 730, 522, 626, 626, 522, 522, 626, 626,
                                            626, 522, 522, 522, 522, 522, 522, 522, 522};
__constant__ double c_min_z[kNPairs] = {-20., 0., -30., -22., 10., -30., -70., -70., -22., 15.,
                                        -30., -70., -70., -20., -22., 0., -30., -70., -70.};
__constant__ double c_max_z[kNPairs] = {20., 30., 0., 22., 30., -10., 70., 70., 22., 30.,
                                        -15., 70., 70., 20., 22., 30., 0., 70., 70.};
__constant__ float c_max_rf[kNPairs] = {20.f, 9.f, 9.f, 20.f, 7.f, 7.f, 5.f, 5.f, 20.f, 6.f, 6.f,
                                        5.f, 5.f, 20.f, 20.f, 9.f, 9.f, 9.f, 9.f};

// CA parameters (ca_hit_ntuplet_generator.jl:9-30), Float32 as Params stores them; the others in alignment.cuh
constexpr float kHardCurv = 0.0328407224959f;
constexpr float kDcaInner = 0.15000000596f;
constexpr float kDcaOuter = 0.25f;

__device__ __forceinline__ uint32_t phi_bin(int16_t t) { return (uint32_t(int32_t(t >> 9)) & 127u) + 1u; }

struct HitView {
  const float *xg, *yg, *zg, *rg;
  const int16_t *iphi, *ysize, *detind;
};

// ---------------------------------------------------------------- doublets
// Block 0, per event: cumulative inner-layer sizes over the pairs and the number of work items, with
// their scan. The other blocks clear what the kernels of the stage count in: the cells ending on each
// hit (the per-cell counters are cleared by the doublet fill that writes the cells), the pools and lists.
__global__ void __launch_bounds__(1024) k_items(Dev d, uint32_t* pair_cum) {
  pdl_sync(d);
  if (blockIdx.x > 0) {
    const uint32_t i0 = (blockIdx.x - 1) * blockDim.x + threadIdx.x, stride = (gridDim.x - 1) * blockDim.x;
    const uint32_t nh = d.ev[d.E].n_hits;
    for (uint32_t i = i0; i < nh; i += stride) d.ohc_cur[i] = 0;
    for (uint32_t i = i0; i < uint32_t(kTpParts); i += stride) d.tp_ctr[i * kTpStride] = 0;
    if (i0 == 0) {
      d.tp_ctr[kTpParts * kTpStride] = 0;
      *d.dbl_pool_ctr = 0;
      *d.cn_pair_ctr = 0;
      d.long_ctr[0] = 0;
      d.long_ctr[1] = 0;
    }
    return;
  }
  __shared__ uint32_t sh[33];
  uint32_t carry = 0;
  for (int b = 0; b < d.E; b += blockDim.x) {
    const int e = b + threadIdx.x;
    uint32_t n = 0;
    if (e < d.E) {
      const uint32_t* hls = d.hits_layer_start + size_t(e) * 11;
      uint32_t acc = 0;
      for (int p = 0; p < kNPairs; ++p) {
        const int li = c_layer_pairs[2 * p];
        acc += hls[li + 1] - hls[li];
        pair_cum[size_t(e) * kNPairs + p] = acc;
      }
      n = d.ev[e].n_hits ? acc : 0u;
    }
    uint32_t tot;
    const uint32_t lo = carry + block_excl_scan(n, sh, &tot);
    if (e < d.E) { d.ev[e].n_items = n; d.ev[e].item_base = lo; }
    carry += tot;
  }
  if (threadIdx.x == 0) { d.ev[d.E].n_items = carry; d.ev[d.E].item_base = carry; }
}

// layer pair and event-local 0-based inner hit of work item j
__device__ __forceinline__ int item_pair(uint32_t j, const uint32_t* cum, const uint32_t* hls, uint32_t* hit) {
  int pid = 0;
  while (j >= cum[pid]) ++pid;
  *hit = ((pid == 0) ? j : j - cum[pid - 1]) + hls[c_layer_pairs[2 * pid]];
  return pid;
}

// Inner-hit part of one work item (inner hit x layer pair): the inner-hit cuts and the
// outer-layer candidates of the phi window, the bins kl .. kh-1 (wrapping after 128) in the
// reference's loop order, which are at most two contiguous ranges of the binned hits.
struct ItemHead {
  float z, r;
  int16_t iphi, ysize, cut;
  uint8_t pid, ok;
  uint32_t hit;             // event-local 0-based inner hit
  uint32_t lo0, n0, lo1;    // candidates: [lo0, lo0 + n0) then [lo1, lo1 + n - n0)
  uint32_t n;
};

__device__ __forceinline__ ItemHead item_head(uint32_t j, const uint32_t* cum, const uint32_t* hls, const HitView& hv,
                                              const uint32_t* poff) {
  ItemHead h{};
  uint32_t i;
  const int pid = item_pair(j, cum, hls, &i);
  h.pid = uint8_t(pid);
  h.hit = i;
  const int inner = c_layer_pairs[2 * pid], outer = c_layer_pairs[2 * pid + 1];
  if (hv.detind[i] > 2000) return h;
  const float me_z = hv.zg[i];
  if (double(me_z) < c_min_z[pid] || double(me_z) > c_max_z[pid]) return h;
  const int32_t me_s = hv.ysize[i];  // idealConditions: every ladder is an outer ladder
  if ((inner == 0 && outer > 3) && (me_s > 0 && me_s < 36)) return h;
  if ((inner == 1 && outer > 3) && (me_s > 0 && me_s < 28)) return h;
  h.ok = 1;
  h.z = me_z;
  h.r = hv.rg[i];
  h.iphi = hv.iphi[i];
  h.ysize = int16_t(me_s);
  h.cut = c_phi_cuts[pid];
  const uint32_t h_off = 128u * uint32_t(outer);
  const uint32_t kl = phi_bin(int16_t(h.iphi - h.cut));
  uint32_t kh = phi_bin(int16_t(h.iphi + h.cut)) + 1;
  if (kh == 129) kh = 1;
  if (kl == kh) return h;
  if (kl < kh) {
    h.lo0 = poff[kl + h_off - 1];
    h.n0 = poff[kh - 1 + h_off] - h.lo0;
    h.lo1 = 0;
    h.n = h.n0;
  } else {
    h.lo0 = poff[kl + h_off - 1];
    h.n0 = poff[128 + h_off] - h.lo0;
    h.lo1 = poff[h_off];
    h.n = h.n0 + (poff[kh - 1 + h_off] - h.lo1);
  }
  return h;
}

// The same item for the count pass, over the binned records sorted by iphi (as uint16) within
// each bin: its candidates are exactly the outer hits that pass the reference's dphi cut
// (|int16(iphi_o - iphi_i)| <= cut), i.e. the part of bin kl from iphi - cut on, the bins
// between, and the part of the last bin up to iphi + cut (two binary searches in the edge bins),
// as at most two ranges when the window wraps past bin 128. The window (2 cut + 1 < 2^15) never
// covers all 128 bins, the reference's kl == kh case.
__device__ __forceinline__ ItemHead item_head_s(uint32_t j, const uint32_t* cum, const uint32_t* hls,
                                                const HitView& hv, const uint32_t* poff, const uint16_t* __restrict__ us) {
  ItemHead h = item_head(j, cum, hls, hv, poff);
  if (!h.ok || h.n == 0) return h;
  const int outer = c_layer_pairs[2 * h.pid + 1];
  const uint32_t h_off = 128u * uint32_t(outer);
  const uint16_t lo_u = uint16_t(h.iphi - h.cut), hi_u = uint16_t(h.iphi + h.cut);
  const uint32_t kl = (uint32_t(lo_u) >> 9) + 1u, km = (uint32_t(hi_u) >> 9) + 1u;  // first, last bin
  uint32_t a = poff[kl - 1 + h_off], ae = poff[kl + h_off];
  while (a < ae) {  // first entry of bin kl at or above lo_u
    const uint32_t m = (a + ae) >> 1;
    if (us[m] < lo_u) a = m + 1; else ae = m;
  }
  uint32_t b = poff[km - 1 + h_off], be = poff[km + h_off];
  while (b < be) {  // one past the last entry of bin km at or below hi_u
    const uint32_t m = (b + be) >> 1;
    if (us[m] <= hi_u) b = m + 1; else be = m;
  }
  if (kl <= km) {
    h.lo0 = a;
    h.n0 = b - a;
    h.lo1 = 0;
    h.n = h.n0;
  } else {
    h.lo0 = a;
    h.n0 = poff[128 + h_off] - a;
    h.lo1 = poff[h_off];
    h.n = h.n0 + (b - h.lo1);
  }
  return h;
}

// The outer-hit cuts of one candidate (gpu_pixel_doublets.jl), in the reference's order:
// doublet_pass_a takes the module, z0 and dphi cuts (about a quarter of the candidates pass),
// doublet_pass_b the cluster-size and pt cuts. c_max_r holds small integers, so the float
// comparison with them equals the reference's Float64 one.
__device__ __forceinline__ bool doublet_pass_a(int pid, float me_z, float me_r, int16_t me_p, int16_t cut,
                                               const HitRec& hr) {
  if (hr.det() > 2000) return false;
  const float dr = __fsub_rn(hr.r, me_r);
  if (dr > c_max_rf[pid] || dr < 0 ||
      fabsf(__fsub_rn(__fmul_rn(me_z, hr.r), __fmul_rn(me_r, hr.z))) > __fmul_rn(12.f, dr))
    return false;
  const int16_t dphi = int16_t(hr.iphi - me_p);
  const int16_t i_dphi = int16_t(dphi < 0 ? -dphi : dphi);
  return i_dphi <= cut;
}

__device__ __forceinline__ bool doublet_pass_b(int pid, float me_z, float me_r, int16_t me_p, int32_t me_s,
                                               const HitRec& hr) {
  const int inner = c_layer_pairs[2 * pid], outer = c_layer_pairs[2 * pid + 1];
  const float dz_dr_fact = float(8 * 0.0285 / 0.015);
  const double min_radius = 0.5 * 87.78;
  const double r2t4 = 4. * min_radius * min_radius;
  const float zo = hr.z, ro = hr.r;
  {  // z_size_cut
    if (outer < 4) {
      const int16_t so = hr.ysize;
      const int dy = inner == 0 ? 28 : 20;
      const int16_t ds = int16_t(so - int16_t(me_s));
      if (me_s > 0 && so > 0 && (ds < 0 ? -int(ds) : int(ds)) > dy) return false;
    } else if (inner < 4 && me_s > 0) {
      const float t = __fmul_rn(fabsf(__fdiv_rn(__fsub_rn(me_z, zo), __fsub_rn(me_r, ro))), dz_dr_fact);
      const double tt = __dadd_rn(double(t), 0.5);
      if (!isfinite(tt)) return false;  // the reference raises (InexactError) here
      const long long pred = (long long)trunc(tt);
      const long long df = (long long)me_s - pred;
      if ((df < 0 ? -df : df) > 20) return false;
    }
  }
  {  // pt_cut
    const int16_t dphi = int16_t(hr.iphi - me_p);
    const int16_t i_dphi = int16_t(dphi < 0 ? -dphi : dphi);
    const double dphi_f = __dmul_rn(double(i_dphi), (2 * 3.141592653589793) / double(1 << 16));
    const float rr = __fmul_rn(me_r, ro);
    const float dd = __fsub_rn(ro, me_r);
    if (__dmul_rn(__dmul_rn(dphi_f, dphi_f), __dsub_rn(r2t4, double(rr))) > double(__fmul_rn(dd, dd))) return false;
  }
  return true;
}

// doublet_pass_a without the dphi cut, for candidates that pass it by construction, and without the
// module's, which the few that pass here take afterwards
__device__ __forceinline__ bool doublet_pass_z(float max_r, float me_z, float me_r, float r, float z) {
  const float dr = __fsub_rn(r, me_r);
  return !(dr > max_r || dr < 0 ||
           fabsf(__fsub_rn(__fmul_rn(me_z, r), __fmul_rn(me_r, z))) > __fmul_rn(12.f, dr));
}

// Reference order of a passing outer hit among its item's cells: the window's bins in order
// (bin offset from the item's first bin kl), then decreasing hit id within a bin. A window of
// at most 2 * 730 + 1 iphi units touches at most four 512-unit bins, so the bin offset takes
// bits 21-26 and bits 27-31 stay free for the item's slot in its warp group (kOwnerShift).
constexpr uint32_t kOwnerShift = 27;
static_assert(kHitIdBits + 6 <= kOwnerShift, "bin offset bits");
__device__ __forceinline__ uint32_t cell_order_key(int16_t me_p, int16_t cut, const HitRec& hr) {
  const uint32_t kl = (uint32_t(uint16_t(me_p - cut)) >> 9) + 1u;
  const uint32_t bo = (((uint32_t(uint16_t(hr.iphi)) >> 9) + 1u - kl) & 127u);
  return (bo << kHitIdBits) | ((kMaxHitsPerEvent - 1u) - hr.id());
}
__device__ __forceinline__ uint32_t key_hit(uint32_t key) { return (kMaxHitsPerEvent - 1u) - (key & (kMaxHitsPerEvent - 1u)); }

__device__ __forceinline__ bool doublet_pass(const ItemHead& h, const HitRec& hr) {
  return doublet_pass_a(h.pid, h.z, h.r, h.iphi, h.cut, hr) && doublet_pass_b(h.pid, h.z, h.r, h.iphi, h.ysize, hr);
}

__device__ __forceinline__ uint32_t head_candidate(const ItemHead& h, uint32_t k) {
  return k < h.n0 ? h.lo0 + k : h.lo1 + (k - h.n0);
}

// All doublets of one item written from event-local position cell_pos on (the fill of
// groups whose count pass could not keep their outer hits).
__device__ __forceinline__ void write_item_doublets(const Dev& d, const ItemHead& h, const HitRec* __restrict__ hrec,
                                                    uint64_t cell_pos, uint64_t cell_lo, uint32_t cap, uint32_t hb) {
  if (!h.ok) return;
  uint32_t cnt = 0;
  for (uint32_t k = 0; k < h.n; ++k) {
    const HitRec hr = hrec[head_candidate(h, k)];
    if (!doublet_pass(h, hr)) continue;
    const uint64_t local = cell_pos + cnt;
    if (local < cap) {
      const uint64_t g = cell_lo + local;
      d.cell_inner[g] = h.hit;
      d.cell_outer[g] = hr.id();
      atomicAdd(&d.ohc_cur[hb + hr.id()], 1u);
      d.cell_pair[g] = h.pid;
      d.cell_id[g] = int32_t(local + 1);
      d.cell_used[g] = 0;
      d.cn_cur[g] = 0;
      d.ct_cur[g] = 0;
    }
    ++cnt;
  }
}

constexpr uint32_t kNoPool = 0xffffffffu;

// Count pass over groups of 32 consecutive items (one warp). The candidates of the group's
// items are laid end to end and take the first cuts 32 at a time on all lanes; the survivors
// (about a quarter) queue in candidate order and take the remaining cuts on full warps, oldest
// first, so passing candidates come out in the order of the cells (item, then the reference's
// candidate order). Their outer hits are staged in shared memory; the group then takes one
// contiguous range of the pool and copies them there. When the staging is nearly full, the items whose
// doublets are complete go to the pool and the current item's move to the front (groups above 768
// doublets are common from pileup 100 on; the fill pass, which searches again what the count could not
// keep, item by item, took 1.48 ms for 111 uneven events). An item that fills the staging alone and the ones
// after it in the group (doublet_staging.cuh), or a full pool, record kNoPool and the fill pass searches again. Bound by
// instructions issued (75 % of the cycles at 300 events of pileup 50); with the first cut's constants staged per
// item and the module cut left to the survivors 512 events take 1.37 ms, before 1.44.
constexpr int kDblQueue = 64;

template <bool kQ>
__global__ void __launch_bounds__(256, 5) k_doublets_count(Dev d, const uint32_t* __restrict__ pair_cum, WorkQueue q) {
  pdl_sync(d);
  __shared__ uint32_t s_cum[kNPairs];
  __shared__ uint32_t s_hls[11];
  // per compacted item: its candidate t is hit record t + x for t < y, t + z from there on; w the pair's
  // largest dr (float bits)
  __shared__ uint4 s_rng[8][32];
  __shared__ uint4 s_geo[8][32];   // per compacted item: z, r (float bits), iphi | cut << 16, pid | ysize << 16
  __shared__ uint16_t s_beg[8][32], s_end[8][32];
  __shared__ uint32_t s_over[8][32];
  __shared__ uint32_t s_q[8][kDblQueue];  // owner << kHitIdBits | candidate
  __shared__ uint32_t s_out[8][kGroupCells];  // owner << kOwnerShift | cell_order_key
  for_each_vblock<kQ>(q, [&](int e, uint32_t bx, uint32_t nbx) {
  const EvInfo& E = d.ev[e];
  const uint32_t n = E.n_items;
  if (n == 0) return;
  if (threadIdx.x < kNPairs) s_cum[threadIdx.x] = pair_cum[size_t(e) * kNPairs + threadIdx.x];
  if (threadIdx.x < 11) s_hls[threadIdx.x] = d.hits_layer_start[size_t(e) * 11 + threadIdx.x];
  __syncthreads();
  const uint32_t hb = E.hit_base;
  HitView hv{d.xg + hb, d.yg + hb, d.zg + hb, d.rg + hb, d.iphi + hb, d.ysize + hb, d.detind + hb};
  const uint32_t* poff = d.phi_off + size_t(e) * kPhiTotBins;
  const HitRec* hrec = d.hit_rec_s + hb;  // sorted by iphi within each bin
  const uint16_t* us = d.hit_u_s + hb;
  const uint32_t ib = E.item_base;
  const unsigned lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
  const unsigned lt = (1u << lane) - 1u;
  for (uint32_t j0 = bx * blockDim.x + 32u * w; j0 < n; j0 += nbx * blockDim.x) {
    const uint32_t j = j0 + lane;
    ItemHead h{};
    if (j < n) h = item_head_s(j, s_cum, s_hls, hv, poff, us);
    const uint32_t nc = h.ok ? h.n : 0u;
    // items with candidates, compacted (compact index = rank among them); the candidates
    // of compacted item c start at position ctex
    const uint32_t busy = __ballot_sync(0xffffffffu, nc > 0);
    const uint32_t ci = __popc(busy & lt);
    const uint32_t ctex = warp_incl_scan(nc) - nc;
    const uint32_t total = __shfl_sync(0xffffffffu, ctex + nc, 31);
    if (nc > 0) {
      s_rng[w][ci] = make_uint4(h.lo0 - ctex, ctex + h.n0, h.lo1 - h.n0 - ctex, __float_as_uint(c_max_rf[h.pid]));
      s_geo[w][ci] = make_uint4(__float_as_uint(h.z), __float_as_uint(h.r),
                                uint32_t(uint16_t(h.iphi)) | (uint32_t(uint16_t(h.cut)) << 16),
                                uint32_t(h.pid) | (uint32_t(uint16_t(h.ysize)) << 16));
    }
    s_over[w][lane] = 0;
    __syncwarp();
    uint32_t nout = 0, qhead = 0, qtail = 0;
    // remaining cuts on queue entries qhead .. qhead + mm - 1, one per lane, in queue order
    auto stage_b = [&](uint32_t mm) {
      bool pass = false;
      uint32_t o = 0, oi = 0;
      if (lane < mm) {
        const uint32_t v = s_q[w][(qhead + lane) % kDblQueue];
        o = v >> kHitIdBits;
        const uint4 g = s_geo[w][o];
        const HitRec hr = hrec[v & (kMaxHitsPerEvent - 1u)];
        pass = hr.det() <= 2000 && doublet_pass_b(int(g.w & 0xffu), __uint_as_float(g.x), __uint_as_float(g.y),
                                                  int16_t(g.z & 0xffffu), int16_t(g.w >> 16), hr);
        oi = (o << kOwnerShift) | cell_order_key(int16_t(g.z & 0xffffu), int16_t(g.z >> 16), hr);
      }
      const uint32_t bal = __ballot_sync(0xffffffffu, pass);
      if (pass) {
        const uint32_t pos = nout + __popc(bal & lt);
        if (pos < uint32_t(kGroupCells)) s_out[w][pos] = oi;
        else atomicAdd(&s_over[w][o], 1u);
      }
      nout += __popc(bal);
      qhead += mm;
    };
    const uint32_t start = nc > 0 ? ctex : 0xffffffffu;
    int cur = -1;       // compacted item owning the candidate before the step
    uint32_t done = 0;  // compacted items whose doublets have gone to the pool
    for (uint32_t t0 = 0;; t0 += 32) {
      const bool last = t0 >= total;
      if (!last) {
        const uint32_t starts = __reduce_or_sync(0xffffffffu, start - t0 < 32u ? 1u << (start - t0) : 0u);
        const uint32_t t = t0 + lane;
        const uint32_t o = uint32_t(cur + int(__popc(starts & ((lt << 1) | 1u))));
        cur += int(__popc(starts));
        bool pass = false;
        uint32_t p = 0;
        if (t < total) {
          const uint4 rg = s_rng[w][o];
          const uint4 g = s_geo[w][o];
          p = t + (t < rg.y ? rg.x : rg.z);
          const float2 zr = *reinterpret_cast<const float2*>(hrec + p);  // z, r
          pass = doublet_pass_z(__uint_as_float(rg.w), __uint_as_float(g.x), __uint_as_float(g.y), zr.y, zr.x);
        }
        const uint32_t bal = __ballot_sync(0xffffffffu, pass);
        if (pass) s_q[w][(qtail + __popc(bal & lt)) % kDblQueue] = (o << kHitIdBits) | p;
        qtail += __popc(bal);
        __syncwarp();
      }
      if (last || qtail - qhead >= 32) {
        stage_b(last ? qtail - qhead : 32u);
        __syncwarp();
      }
      if (!last && !staging_near_full(nout)) continue;
      // the staged outputs are in item order, so each item's are one run; the items before `keep` are complete
      const uint32_t nst = nout < uint32_t(kGroupCells) ? nout : uint32_t(kGroupCells);
      const uint32_t keep = last ? 32u : s_out[w][nst - 1] >> kOwnerShift;
      if (!last && !staging_hands_over(nout, keep, done)) continue;
      s_beg[w][lane] = 0; s_end[w][lane] = 0;
      __syncwarp();
      for (uint32_t x = lane; x < nst; x += 32) {
        const uint32_t o = s_out[w][x] >> kOwnerShift;
        if (x == 0 || (s_out[w][x - 1] >> kOwnerShift) != o) s_beg[w][o] = uint16_t(x);
        if (x + 1 == nst || (s_out[w][x + 1] >> kOwnerShift) != o) s_end[w][o] = uint16_t(x + 1);
      }
      __syncwarp();
      const bool mine = nc > 0 ? ci >= done && ci < keep : last;
      const uint32_t cnt = mine && nc > 0 ? s_end[w][ci] - s_beg[w][ci] + s_over[w][ci] : 0u;
      const uint32_t ncopy = last ? nst : s_beg[w][keep];
      if (mine && j < n) d.item_cnt[ib + j] = cnt;
      uint32_t off = kNoPool;
      if (nout > 0 && nout <= uint32_t(kGroupCells)) {
        uint32_t o = 0;
        if (lane == 0) o = atomicAdd(d.dbl_pool_ctr, ncopy);
        o = __shfl_sync(0xffffffffu, o, 0);
        if (uint64_t(o) + ncopy <= uint64_t(d.cap_cells)) off = o;
      }
      // each staged outer hit goes to its place in the reference's cell order, its rank by key
      // among its item's (they came in iphi order within each bin)
      if (off != kNoPool)
        for (uint32_t x = lane; x < ncopy; x += 32) {
          const uint32_t v = s_out[w][x];
          const uint32_t b0 = s_beg[w][v >> kOwnerShift], b1 = s_end[w][v >> kOwnerShift];
          uint32_t rank = 0;
          for (uint32_t y = b0; y < b1; ++y) rank += s_out[w][y] < v;
          d.dbl_pool[off + b0 + rank] = key_hit(v);
        }
      const uint32_t ex = warp_incl_scan(cnt) - cnt;
      if (mine && j < n) d.item_pool[ib + j] = off == kNoPool ? kNoPool : off + ex;
      __syncwarp();
      if (last) break;
      for (uint32_t x0 = ncopy; x0 < nout; x0 += 32) {  // the current item's doublets to the front
        const uint32_t v = x0 + lane < nout ? s_out[w][x0 + lane] : 0u;
        __syncwarp();
        if (x0 + lane < nout) s_out[w][x0 - ncopy + lane] = v;
        __syncwarp();
      }
      nout -= ncopy;
      done = keep;
    }
  }
  });
}

// Fill pass over the same 32-item groups: cells of a group are contiguous, so the warp
// writes them with consecutive lanes on consecutive cells, outer hits from the pool and the
// inner hit and pair of each cell's item from shared memory. Bound by its 22 bytes of stores and one
// atomic per cell; the items that own a step's cells come from a bit mask (with a binary search per cell 512
// events of pileup 50 took 474 us, now 457; one of pileup 170 45 and 40).
template <bool kQ>
__global__ void __launch_bounds__(256) k_doublets_fill(Dev d, const uint32_t* __restrict__ pair_cum, WorkQueue q) {
  pdl_sync(d);
  __shared__ uint32_t s_cum[kNPairs];
  __shared__ uint32_t s_hls[11];
  // of the items with doublets: where the item's pool range would put the group's cell 0, its hit, its pair
  __shared__ uint4 s_item[8][32];
  for_each_vblock<kQ>(q, [&](int e, uint32_t bx, uint32_t nbx) {
  const EvInfo& E = d.ev[e];
  const uint32_t n = E.n_items;
  if (n == 0) return;
  if (threadIdx.x < kNPairs) s_cum[threadIdx.x] = pair_cum[size_t(e) * kNPairs + threadIdx.x];
  if (threadIdx.x < 11) s_hls[threadIdx.x] = d.hits_layer_start[size_t(e) * 11 + threadIdx.x];
  __syncthreads();
  const uint32_t hb = E.hit_base;
  HitView hv{d.xg + hb, d.yg + hb, d.zg + hb, d.rg + hb, d.iphi + hb, d.ysize + hb, d.detind + hb};
  const uint32_t* poff = d.phi_off + size_t(e) * kPhiTotBins;
  const HitRec* hrec = d.hit_rec + hb;
  const uint32_t ib = E.item_base;
  // raw positions of the count scan are made local to the event; the event keeps its
  // first n_cells doublets, stored from cell_base on
  const uint32_t raw_lo = d.item_cnt[ib];
  const uint64_t cell_lo = E.cell_base;
  const uint32_t keep = E.n_cells;
  const unsigned lane = threadIdx.x & 31u, w = threadIdx.x >> 5, lt = (1u << lane) - 1u;
  for (uint32_t j0 = bx * blockDim.x + 32u * w; j0 < n; j0 += nbx * blockDim.x) {
    const uint32_t j = j0 + lane;
    const bool valid = j < n;
    const uint32_t pos = valid ? d.item_cnt[ib + j] - raw_lo : 0u;
    const uint32_t cnt = valid ? d.item_cnt[ib + j + 1] - d.item_cnt[ib + j] : 0u;
    const uint32_t pool = valid ? d.item_pool[ib + j] : kNoPool;
    if (__any_sync(0xffffffffu, cnt > 0 && pool == kNoPool)) {
      if (cnt > 0) write_item_doublets(d, item_head(j, s_cum, s_hls, hv, poff), hrec, pos, cell_lo, keep, hb);
      continue;
    }
    const uint32_t inc = warp_incl_scan(cnt);
    const uint32_t total = __shfl_sync(0xffffffffu, inc, 31);
    if (total == 0) continue;
    const uint32_t base = __shfl_sync(0xffffffffu, pos, 0);
    uint32_t i = 0;
    const int pid = valid ? item_pair(j, s_cum, s_hls, &i) : 0;
    const uint32_t busy = __ballot_sync(0xffffffffu, cnt > 0);
    if (cnt > 0) s_item[w][__popc(busy & lt)] = make_uint4(pool - (inc - cnt), i, uint32_t(pid), 0);
    __syncwarp();
    const uint32_t start = cnt > 0 ? inc - cnt : 0xffffffffu;
    const uint32_t m = base < keep ? min(total, keep - base) : 0u;
    int cur = -1;  // item owning the cell before the step
    for (uint32_t x0 = 0; x0 < m; x0 += 32) {
      const uint32_t starts = __reduce_or_sync(0xffffffffu, start - x0 < 32u ? 1u << (start - x0) : 0u);
      const uint32_t a = uint32_t(cur + int(__popc(starts & ((lt << 1) | 1u))));
      cur += int(__popc(starts));
      const uint32_t x = x0 + lane;
      if (x >= m) continue;
      const uint4 it = s_item[w][a];
      const uint64_t g = cell_lo + base + x;
      d.cell_inner[g] = it.y;
      const uint32_t oh = d.dbl_pool[it.x + x];
      d.cell_outer[g] = oh;
      atomicAdd(&d.ohc_cur[hb + oh], 1u);  // cells ending on each hit
      d.cell_pair[g] = uint8_t(it.z);
      d.cell_id[g] = int32_t(base + x + 1);
      d.cell_used[g] = 0;
      d.cn_cur[g] = 0;
      d.ct_cur[g] = 0;
    }
    __syncwarp();
  }
  });
}

// per event: capped doublet count, its scan into the cell bases, and events past the cell buffer
// emptied (as k_ev_scan does it); one block
__global__ void __launch_bounds__(1024) k_cell_bases(Dev d) {
  pdl_sync(d);
  __shared__ uint32_t sh[33];
  uint32_t carry = 0;
  for (int b = 0; b < d.E; b += blockDim.x) {
    const int e = b + threadIdx.x;
    uint32_t n = 0;
    if (e < d.E) {
      EvInfo& E = d.ev[e];
      n = d.item_cnt[E.item_base + E.n_items] - d.item_cnt[E.item_base];
      E.n_cols_nb = 0;
      E.n_cols_tr = 0;
      // the reference keeps the first doublets_per_event
      if (n > d.doublets_per_event) { n = d.doublets_per_event; E.warnings |= kWarnDoublets; }
    }
    uint32_t tot;
    const uint32_t lo = carry + block_excl_scan(n, sh, &tot);
    if (e < d.E) {
      EvInfo& E = d.ev[e];
      if (int64_t(lo) + int64_t(n) > d.cap_cells) {
        n = 0;
        E.warnings |= kWarnBuffer;
        atomicOr(d.status, kWarnBuffer);
      }
      E.cell_base = lo;
      E.n_cells = n;
      E.n_cells_raw = n;
    }
    carry += tot;
  }
  if (threadIdx.x == 0) {
    EvInfo& T = d.ev[d.E];
    T.cell_base = carry;
    T.n_cells = int64_t(carry) > d.cap_cells ? uint32_t(d.cap_cells) : carry;
    T.n_cells_raw = T.n_cells;
  }
}

// ---------------------------------------------------------------- outer-hit lists
// cells ending on each hit: slots from the shifted scan of the counts the doublet fill took
constexpr int kOhcUnroll = 4;  // cells (list entries) per thread and step, loads independent

__global__ void k_ohc_fill(Dev d) {
  pdl_sync(d);
  const int e = blockIdx.y;
  const EvInfo& E = d.ev[e];
  const uint64_t cb = E.cell_base;
  const uint32_t hb = E.hit_base;
  const uint32_t n = E.n_cells, stride = gridDim.x * blockDim.x;
  for (uint32_t k0 = blockIdx.x * blockDim.x + threadIdx.x; k0 < n; k0 += kOhcUnroll * stride) {
    uint32_t o[kOhcUnroll], slot[kOhcUnroll];
#pragma unroll
    for (int u = 0; u < kOhcUnroll; ++u) o[u] = k0 + u * stride < n ? d.cell_outer[cb + k0 + u * stride] : 0xffffffffu;
#pragma unroll
    for (int u = 0; u < kOhcUnroll; ++u)
      if (o[u] != 0xffffffffu) slot[u] = atomicAdd(&d.ohc_cnt[hb + o[u] + 1], 1u);
#pragma unroll
    for (int u = 0; u < kOhcUnroll; ++u)
      if (o[u] != 0xffffffffu) d.ohc_list[slot[u]] = uint32_t(cb + k0 + u * stride);
  }
}

// bitonic sorting network over N values held in registers (indices are compile-time)
template <int N>
__device__ __forceinline__ void bitonic_regs(uint32_t (&v)[N]) {
#pragma unroll
  for (int k = 2; k <= N; k <<= 1) {
#pragma unroll
    for (int j = k >> 1; j > 0; j >>= 1) {
#pragma unroll
      for (int i = 0; i < N; ++i) {
        const int l = i ^ j;
        if (l > i) {
          const uint32_t lo = min(v[i], v[l]), hi = max(v[i], v[l]);
          if ((i & k) == 0) { v[i] = lo; v[l] = hi; } else { v[i] = hi; v[l] = lo; }
        }
      }
    }
  }
}

template <int N>
__device__ __forceinline__ void sort_regs(uint32_t* a, uint32_t n) {
  uint32_t v[N];
#pragma unroll
  for (int i = 0; i < N; ++i) v[i] = uint32_t(i) < n ? a[i] : 0xffffffffu;  // padding sorts last
  bitonic_regs<N>(v);
#pragma unroll
  for (int i = 0; i < N; ++i)
    if (uint32_t(i) < n) a[i] = v[i];
}

// Sorts a list of at most kMax entries in place with a register network and returns true;
// longer lists are left to k_sort_long (a list kernel keeps the few registers of its largest
// network, which sets its occupancy).
template <int kMax>
__device__ __forceinline__ bool sort_short(uint32_t* a, uint32_t n) {
  if (n < 2) return true;
  if (n <= 4) { sort_regs<4>(a, n); return true; }
  if (n <= 8) { sort_regs<8>(a, n); return true; }
  return false;
}

__device__ __forceinline__ void insertion_sort(uint32_t* a, uint32_t n) {
  for (uint32_t p = 1; p < n; ++p) {
    const uint32_t v = a[p];
    uint32_t q = p;
    while (q > 0 && a[q - 1] > v) { a[q] = a[q - 1]; --q; }
    a[q] = v;
  }
}

// sort a short list in place (ascending; entries are ids below 0xffffffff): one load and
// one store per entry through a register network up to 32 entries, insertion sort above
__device__ __forceinline__ void sort_list(uint32_t* a, uint32_t n) {
  if (n < 2) return;
  if (n <= 4) { sort_regs<4>(a, n); return; }
  if (n <= 8) { sort_regs<8>(a, n); return; }
  if (n <= 16) { sort_regs<16>(a, n); return; }
  if (n <= 32) { sort_regs<32>(a, n); return; }
  insertion_sort(a, n);
}

// lists above the short-sort limit, sorted afterwards by k_sort_long (a list of n entries
// needs n > 8, so the buffer of cap_long = entries / 9 entries cannot overflow)
__device__ __forceinline__ void push_long_list(const Dev& d, int kind, uint32_t lo, uint32_t n) {
  const uint32_t slot = atomicAdd(&d.long_ctr[kind], 1u);
  if (slot < uint32_t(d.cap_long)) d.long_lists[slot] = make_uint2(lo, n);
  else atomicOr(d.status, kWarnBuffer);
}

constexpr int kSortLongBlocks = 148 * 4;

__global__ void __launch_bounds__(256) k_sort_long(Dev d, int kind, uint32_t* list) {
  pdl_sync(d);
  uint32_t nl = d.long_ctr[kind];
  if (nl > uint32_t(d.cap_long)) nl = uint32_t(d.cap_long);
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nl; i += gridDim.x * blockDim.x) {
    const uint2 l = d.long_lists[i];
    sort_list(list + l.x, l.y);
  }
}

// Sorts the outer-hit lists (ascending) and gathers connect's candidate of each entry. A warp takes
// `hits` consecutive hits, fewer than 32 in a small batch. Their lists lie end to end: as many whole lists
// as fit are staged, a lane takes an entry, and its place is the number of entries of its list that are
// below it (entries differ). Reads and writes stay on the region's lines; a lane per list, with register
// networks by length up to 32 and a warp per longer one, loaded and stored a line per lane and entry (fill,
// sort and gather, the latter in a kernel of its own: 512 events of pileup 50 693 us, 111 of pileup 1 to 200
// 925; now 620 and 615). 512 staged entries per warp: with 1024 the shared memory leaves no L1 (706 and
// 685 us), with 256 more groups are cut (628 and 636). Lists above the staging
// (none at pileup 200, whose longest has 125 entries) are sorted by one lane.
constexpr int kRankBuf = 512;

__global__ void __launch_bounds__(256) k_sort_hit_lists(Dev d, uint32_t hits) {
  pdl_sync(d);
  __shared__ uint32_t s_list[8][kRankBuf];
  __shared__ uint32_t s_beg[8][33];  // first staged entry of each staged list, and one past the last
  const int e = blockIdx.y;
  const EvInfo& E = d.ev[e];
  const uint32_t hb = E.hit_base, nh = E.n_hits;
  const unsigned lane = threadIdx.x & 31u, w = threadIdx.x >> 5, lt = (1u << lane) - 1u;
  const uint32_t warps = gridDim.x * (blockDim.x / 32);
  uint32_t* sl = s_list[w];
  uint32_t* sb = s_beg[w];
  auto put = [&](uint32_t pos, uint32_t cell, uint32_t ih) {
    const float4 h = d.hit_xyzr[hb + ih];
    const int16_t det = d.detind[hb + ih];
    d.ohc_list[pos] = cell;
    d.ohc_rec[pos] = make_float2(det < 96 ? -h.w : h.w, h.z);
  };
  for (uint32_t k0 = (blockIdx.x * (blockDim.x / 32) + w) * hits; k0 < nh; k0 += warps * hits) {
    const uint32_t k = k0 + lane;
    const uint32_t first = d.ohc_cnt[hb + k0];
    uint32_t ex = 0, n = 0;  // first entry of the lane's list from `first` on, entries
    if (lane < hits && k < nh) {
      const uint32_t lo = d.ohc_cnt[hb + k];
      n = d.ohc_cnt[hb + k + 1] - lo;
      ex = lo - first;
      if (n > uint32_t(kMaxCellsPerHit)) atomic_or_warn(&d.ev[e], kWarnLists);
    }
    const uint32_t total = __reduce_max_sync(0xffffffffu, n > 0 ? ex + n : 0u);
    for (uint32_t c0 = 0; c0 < total;) {
      const bool in = n > 0 && ex >= c0 && ex + n <= c0 + uint32_t(kRankBuf);
      const uint32_t m = __ballot_sync(0xffffffffu, in);
      if (m == 0) {  // the next list exceeds the staging
        const bool mine = n > 0 && ex == c0;
        if (mine) {
          insertion_sort(d.ohc_list + first + ex, n);
          for (uint32_t p = first + ex; p < first + ex + n; ++p) put(p, d.ohc_list[p], d.cell_inner[d.ohc_list[p]]);
        }
        c0 += __reduce_max_sync(0xffffffffu, mine ? n : 0u);
        continue;
      }
      const uint32_t len = __reduce_max_sync(0xffffffffu, in ? ex + n - c0 : 0u);
      if (in) sb[__popc(m & lt)] = ex - c0;
      if (lane == 0) sb[__popc(m)] = len;
      for (uint32_t x = lane; x < len; x += 32) sl[x] = d.ohc_list[first + c0 + x];
      __syncwarp();
      const uint32_t start = in ? ex - c0 : 0xffffffffu;
      int cur = -1;
      for (uint32_t x0 = 0; x0 < len; x0 += 32) {
        const uint32_t starts = __reduce_or_sync(0xffffffffu, start - x0 < 32u ? 1u << (start - x0) : 0u);
        const uint32_t a = uint32_t(cur + int(__popc(starts & ((lt << 1) | 1u))));
        cur += int(__popc(starts));
        if (x0 + lane < len) {
          const uint32_t v = sl[x0 + lane];
          const uint32_t ih = d.cell_inner[v];
          const uint32_t b0 = sb[a], b1 = sb[a + 1];
          uint32_t rank = 0;
#pragma unroll 4
          for (uint32_t y = b0; y < b1; ++y) rank += sl[y] < v;
          put(first + c0 + b0 + rank, v, ih);
        }
      }
      __syncwarp();
      c0 += len;
    }
  }
}

// ---------------------------------------------------------------- connect
struct CircleEq {
  float xp, yp, c, alpha, beta;
  __device__ CircleEq(float x1, float y1, float x2, float y2, float x3, float y3) {
    const bool no_flip = fabsf(__fsub_rn(x3, x1)) < fabsf(__fsub_rn(y3, y1));
    const float x1p = no_flip ? __fsub_rn(x1, x2) : __fsub_rn(y1, y2);
    const float y1p = no_flip ? __fsub_rn(y1, y2) : __fsub_rn(x1, x2);
    const float d12 = __fadd_rn(__fmul_rn(x1p, x1p), __fmul_rn(y1p, y1p));
    const float x3p = no_flip ? __fsub_rn(x3, x2) : __fsub_rn(y3, y2);
    const float y3p = no_flip ? __fsub_rn(y3, y2) : __fsub_rn(x3, x2);
    const float d32 = __fadd_rn(__fmul_rn(x3p, x3p), __fmul_rn(y3p, y3p));
    const float num = __fsub_rn(__fmul_rn(x1p, y3p), __fmul_rn(y1p, x3p));
    const float det = __fsub_rn(__fmul_rn(d12, y3p), __fmul_rn(d32, y1p));
    const float st2 = __fsub_rn(__fmul_rn(d12, x3p), __fmul_rn(d32, x1p));
    const float seq = __fadd_rn(__fmul_rn(det, det), __fmul_rn(st2, st2));
    float al2 = __fdiv_rn(1.0f, __fsqrt_rn(seq));
    const float be2 = __fmul_rn(-st2, al2);
    const float ct = __fmul_rn(__fmul_rn(2.0f, num), al2);
    al2 = __fmul_rn(al2, det);
    xp = x2; yp = y2;
    c = no_flip ? ct : -ct;
    alpha = no_flip ? al2 : -be2;
    beta = no_flip ? be2 : -al2;
  }
  __device__ float dca0() const {
    const float x = __fadd_rn(__fmul_rn(c, xp), alpha);
    const float y = __fadd_rn(__fmul_rn(c, yp), beta);
    return __fsub_rn(__fsqrt_rn(__fadd_rn(__fmul_rn(x, x), __fmul_rn(y, y))), 1.0f);
  }
};

// Connection test of every cell with the cells ending on its inner hit (the outer-hit list,
// at most kMaxCellsPerHit entries). A warp takes 32 cells and spreads their (cell, candidate)
// pairs over its lanes, 32 pairs per step; a bound of the alignment test runs on every pair, and the
// pairs that pass it (a few percent) queue in shared memory for that test and the circle / DCA test,
// which then run on full warps: the queue goes on over the warp's cells (emptied after every 32 of
// them, a circle test of 150 instructions ran for five pairs: connect of 512 events of pileup 50
// 1.33 ms, then 1.18; of 111 of pileup 1 to 200, 2.75 and 2.58 ms). Bound by instructions issued (78 % of
// the cycles at 300 events of pileup 50): the test itself with its square root on every pair, and a search for each pair's
// cell in place of the bit mask of the cells that start in a step, took 1.18 and 2.58 ms, now 0.94
// and 2.16. Six blocks per SM (40 registers, two of them spilled) against five: 0.94 and 0.98 ms.
// A passing pair counts one neighbour of the candidate (cn_cur), sets both used flags and goes to the pair list that k_connect_fill turns into neighbour lists; none
// of these depends on the evaluation order.
constexpr int kConnWarps = 8;
constexpr int kConnQueue = 64;

template <bool kQ>
__global__ void __launch_bounds__(256, 6) k_connect_test(Dev d, WorkQueue q) {
  pdl_sync(d);
  // of the cells with candidates: inner r (negative: barrel), z and outer r, z; the cell; the list
  // position of pair 0, were all cells' candidates one list
  __shared__ float4 s_rz[kConnWarps][32];
  __shared__ uint2 s_cell[kConnWarps][32];
  __shared__ uint2 s_queue[kConnWarps][kConnQueue];  // pair: cell, list position of the candidate
  for_each_vblock<kQ>(q, [&](int e, uint32_t bx, uint32_t nbx) {
  const EvInfo& E = d.ev[e];
  const uint64_t cb = E.cell_base;
  const uint32_t hb = E.hit_base;
  const float4* hxyzr = d.hit_xyzr + hb;
  const unsigned lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
  const unsigned lt = (1u << lane) - 1u;
  uint32_t qn = 0;
  // circle / DCA test of the queued pairs q0 .. q0+31 (lanes past qn idle)
  auto circle_step = [&](uint32_t q0, uint32_t qn) {
    bool cut = false;
    uint32_t o = 0, c = 0;
    if (q0 + lane < qn) {
      const uint2 v = s_queue[w][q0 + lane];
      c = v.x;
      o = d.ohc_list[v.y];
      const float region = signbit(d.ohc_rec[v.y].x) ? kDcaInner : kDcaOuter;
      const uint32_t ih = d.cell_inner[c];
      const float4 h1 = hxyzr[d.cell_inner[o]];  // the candidate's inner hit
      const float4 hi = hxyzr[ih], ho = hxyzr[d.cell_outer[c]];
      if (are_aligned(h1.w, h1.z, hi.w, hi.z, ho.w, ho.z, d.detind[hb + ih] < 1184 ? kThetaBarrel : kThetaForward)) {
        const CircleEq eq(h1.x, h1.y, hi.x, hi.y, ho.x, ho.y);
        if (eq.c > kHardCurv) cut = false;
        else cut = fabsf(eq.dca0()) < __fmul_rn(region, fabsf(eq.c));
      }
    }
    const uint32_t bal = __ballot_sync(0xffffffffu, cut);
    if (bal) {
      uint32_t base = 0;
      if (lane == 0) base = atomicAdd(d.cn_pair_ctr, uint32_t(__popc(bal)));
      base = __shfl_sync(0xffffffffu, base, 0);
      if (cut) {
        const uint32_t slot = base + __popc(bal & lt);
        d.cell_used[o] = 1;
        d.cell_used[c] = 1;
        if (slot < uint32_t(d.cap_pairs)) {
          d.cn_pairs[slot] = make_uint2(o, c);
          atomicAdd(&d.cn_cur[o], 1u);
        } else {
          atomicOr(d.status, kWarnBuffer);
        }
      }
    }
  };
  for (uint32_t k0 = bx * blockDim.x + 32u * w; k0 < E.n_cells; k0 += nbx * blockDim.x) {
    const uint32_t k = k0 + lane;
    const uint64_t c = cb + k;
    uint32_t n = 0, lo = 0, ih = 0;
    if (k < E.n_cells) {
      ih = d.cell_inner[c];
      lo = d.ohc_cnt[hb + ih];
      n = d.ohc_cnt[hb + ih + 1] - lo;
      if (n > uint32_t(kMaxCellsPerHit)) n = kMaxCellsPerHit;
    }
    const uint32_t ex = warp_incl_scan(n) - n;
    const uint32_t total = __shfl_sync(0xffffffffu, ex + n, 31);
    const uint32_t busy = __ballot_sync(0xffffffffu, n > 0);
    if (n > 0) {  // geometry only for cells with candidates
      const uint32_t oh = d.cell_outer[c], a = __popc(busy & lt);
      const float4 hi = hxyzr[ih], ho = hxyzr[oh];
      s_rz[w][a] = make_float4(d.detind[hb + ih] < 1184 ? -hi.w : hi.w, hi.z, ho.w, ho.z);
      s_cell[w][a] = make_uint2(uint32_t(c), lo - ex);
    }
    __syncwarp();
    const uint32_t start = n > 0 ? ex : 0xffffffffu;
    int cur = -1;  // owner of the pair before the step
    for (uint32_t x0 = 0; x0 < total; x0 += 32) {
      const uint32_t starts = __reduce_or_sync(0xffffffffu, start - x0 < 32u ? 1u << (start - x0) : 0u);
      const uint32_t a = uint32_t(cur + int(__popc(starts & ((lt << 1) | 1u))));
      cur += int(__popc(starts));
      bool al = false;
      uint2 pair = make_uint2(0, 0);
      if (x0 + lane < total) {
        pair = s_cell[w][a];
        pair.y += x0 + lane;
        const float2 rec = d.ohc_rec[pair.y];  // the candidate's inner hit: r (sign: inner barrel), z
        const float4 rz = s_rz[w][a];
        al = maybe_aligned(fabsf(rec.x), rec.y, fabsf(rz.x), rz.y, rz.z, rz.w, signbit(rz.x));
      }
      const uint32_t bal = __ballot_sync(0xffffffffu, al);
      if (al) s_queue[w][qn + __popc(bal & lt)] = pair;
      qn += __popc(bal);
      __syncwarp();
      if (qn >= 32) {
        qn -= 32;
        circle_step(qn, qn + 32);
        __syncwarp();
      }
    }
    __syncwarp();
  }
  circle_step(0, qn);
  });
}

// neighbour lists from the pair list: each passing (candidate o, cell c) appends c to o's list
__global__ void __launch_bounds__(256) k_connect_fill(Dev d) {
  pdl_sync(d);
  uint32_t np = *d.cn_pair_ctr;
  if (np > uint32_t(d.cap_pairs)) np = uint32_t(d.cap_pairs);
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < np; i += gridDim.x * blockDim.x) {
    const uint2 pc = d.cn_pairs[i];
    d.cn_list[atomicAdd(&d.cn_cnt[pc.x + 1], 1u)] = pc.y;
  }
}

// per-cell lists: neighbours (kind 0) or tracks (kind 1), sorted ascending; flags overflow
template <int kKind>
__global__ void k_sort_cell_lists(Dev d) {
  pdl_sync(d);
  const int e = blockIdx.y;
  const EvInfo& E = d.ev[e];
  const uint64_t cb = E.cell_base;
  __shared__ uint32_t s_cols;
  if (threadIdx.x == 0) s_cols = 0;
  __syncthreads();
  uint32_t cols = 0;
  for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < E.n_cells; k += gridDim.x * blockDim.x) {
    const uint64_t c = cb + k;
    const uint32_t* cnt = kKind == 0 ? d.cn_cnt : d.ct_cnt;
    uint32_t* list = kKind == 0 ? d.cn_list : d.ct_list;
    const uint32_t lo = cnt[c];
    uint32_t hi = cnt[c + 1];
    const uint64_t lcap = uint64_t(kKind == 0 ? d.cap_pairs : d.cap_tuple_hits);
    if (uint64_t(hi) > lcap) hi = uint32_t(lcap);
    if (hi > lo) {
      ++cols;
      if (!sort_short<8>(list + lo, hi - lo)) push_long_list(d, kKind, lo, hi - lo);
      if (hi - lo > uint32_t(kCellRows)) atomic_or_warn(&d.ev[e], kWarnLists);
    }
    // cells with two or more tracks, for the duplicate remover
    if (kKind == 1 && cnt[c + 1] - cnt[c] >= 2) atomicOr(&d.dup_bits[c >> 5], 1u << (c & 31));
  }
  if (cols) atomicAdd(&s_cols, cols);
  __syncthreads();
  if (threadIdx.x == 0 && s_cols) {
    // columns of the fixed column store: one per cell with a non-empty list plus the reserved one
    uint32_t* counter = kKind == 0 ? &d.ev[e].n_cols_nb : &d.ev[e].n_cols_tr;
    const uint32_t before = atomicAdd(counter, s_cols);
    if (before + s_cols + 1 > d.columns_per_event) atomic_or_warn(&d.ev[e], kWarnColumns);
  }
}

// ---------------------------------------------------------------- fishbone
template <bool kQ>
__global__ void __launch_bounds__(128) k_fishbone(Dev d, WorkQueue q) {
  pdl_sync(d);
  for_each_vblock<kQ>(q, [&](int e, uint32_t bx, uint32_t nbx) {
  const EvInfo& E = d.ev[e];
  if (E.n_hits <= 1) return;
  const uint32_t hb = E.hit_base;
  const float* xg = d.xg + hb;
  const float* yg = d.yg + hb;
  const float* zg = d.zg + hb;
  const int16_t* det = d.detind + hb;
  for (uint32_t k = bx * blockDim.x + threadIdx.x; k < E.n_hits; k += nbx * blockDim.x) {
    const uint32_t lo = d.ohc_cnt[hb + k];
    uint32_t n = d.ohc_cnt[hb + k + 1] - lo;
    if (n < 2) continue;
    if (n > uint32_t(kMaxCellsPerHit)) n = kMaxCellsPerHit;
    const uint32_t* L = d.ohc_list + lo;
    const float xo = xg[k], yo = yg[k], zo = zg[k];
    // the cells that carry a neighbour relation, in list order
    float dx[kMaxCellsPerHit], dy[kMaxCellsPerHit], dz[kMaxCellsPerHit], nrm[kMaxCellsPerHit];
    uint16_t idet[kMaxCellsPerHit];
    uint8_t idx[kMaxCellsPerHit];
    // gathered kFishBatch entries at a time: each stage's loads are independent of one
    // another, so a batch waits for four load latencies rather than four per entry
    constexpr int kFishBatch = 8;
    uint32_t curr = 0;
    for (uint32_t j0 = 0; j0 < n; j0 += kFishBatch) {
      uint32_t cb8[kFishBatch], ih8[kFishBatch];
      bool used[kFishBatch];
#pragma unroll
      for (int i = 0; i < kFishBatch; ++i) cb8[i] = j0 + i < n ? L[j0 + i] : 0u;
#pragma unroll
      for (int i = 0; i < kFishBatch; ++i) used[i] = j0 + i < n && d.cell_used[cb8[i]] != 0;
#pragma unroll
      for (int i = 0; i < kFishBatch; ++i) ih8[i] = used[i] ? d.cell_inner[cb8[i]] : 0u;
#pragma unroll
      for (int i = 0; i < kFishBatch; ++i) {
        if (!used[i]) continue;
        const float4 hi = d.hit_xyzr[hb + ih8[i]];
        idx[curr] = uint8_t(j0 + i);
        idet[curr] = uint16_t(det[ih8[i]]);
        dx[curr] = __fsub_rn(hi.x, xo);
        dy[curr] = __fsub_rn(hi.y, yo);
        dz[curr] = __fsub_rn(hi.z, zo);
        nrm[curr] = __fadd_rn(__fadd_rn(__fmul_rn(dx[curr], dx[curr]), __fmul_rn(dy[curr], dy[curr])),
                              __fmul_rn(dz[curr], dz[curr]));
        ++curr;
      }
    }
    if (curr < 2) continue;
    for (uint32_t ic = 0; ic + 1 < curr; ++ic) {
      for (uint32_t jc = ic + 1; jc < curr; ++jc) {
        const float cos12 = __fadd_rn(__fadd_rn(__fmul_rn(dx[ic], dx[jc]), __fmul_rn(dy[ic], dy[jc])),
                                      __fmul_rn(dz[ic], dz[jc]));
        if (idet[ic] != idet[jc] &&
            __fmul_rn(cos12, cos12) >= __fmul_rn(__fmul_rn(0.99999f, nrm[ic]), nrm[jc])) {
          if (nrm[ic] > nrm[jc]) { d.cell_id[L[idx[ic]]] = -1; break; }
          d.cell_id[L[idx[jc]]] = -1;
        }
      }
    }
  }
  });
}

// ---------------------------------------------------------------- ntuplets
constexpr int kMaxDepth = 8;

// Depth-first walk of find_ntuplets from one start cell. kFill == false counts tuples and
// hits and appends each tuple's record (its doublets, and its ordinal and hit offset among the
// start cell's tuples) to part `part` of the record pool; kFill == true writes the tuples from
// the given global tuple / hit positions (run only when the pool overflowed).
template <bool kFill>
__device__ void walk(const Dev& d, uint64_t cb, uint64_t start, uint64_t* tuple_pos, uint64_t* hit_pos,
                     uint32_t* ntup, uint32_t* nhit, uint64_t tuple_lo, uint32_t tcap, int e, uint32_t part) {
  uint32_t stack_c[kMaxDepth];
  uint32_t stack_k[kMaxDepth];
  int depth = 0;
  stack_c[0] = uint32_t(start);
  stack_k[0] = 0;
  bool descended = false;  // whether the current top has an alive neighbour
  bool alive_child[kMaxDepth];
  alive_child[0] = false;
  (void)descended;
  while (depth >= 0) {
    const uint32_t c = stack_c[depth];
    const uint32_t lo = d.cn_cnt[c];
    uint32_t nn = d.cn_cnt[c + 1] - lo;
    if (nn > uint32_t(kCellRows)) nn = kCellRows;
    // entries past the pair buffer were not stored (buffer warning raised by the fill)
    if (uint64_t(lo) + nn > uint64_t(d.cap_pairs)) nn = uint64_t(lo) < uint64_t(d.cap_pairs) ? uint32_t(d.cap_pairs - lo) : 0u;
    bool pushed = false;
    while (stack_k[depth] < nn) {
      const uint32_t o = d.cn_list[lo + stack_k[depth]];
      stack_k[depth]++;
      if (d.cell_id[o] < 0) continue;  // killed by the fishbone
      alive_child[depth] = true;
      if (depth + 1 >= kMaxDepth) { atomic_or_warn(&d.ev[e], kWarnTuples); continue; }
      ++depth;
      stack_c[depth] = o;
      stack_k[depth] = 0;
      alive_child[depth] = false;
      pushed = true;
      break;
    }
    if (pushed) continue;
    // all neighbours of the top visited
    if (!alive_child[depth] && depth >= 1) {
      const uint32_t nh = uint32_t(depth) + 2;  // doublets on the stack + 1
      if (kFill) {
        const uint64_t g = *tuple_pos;
        const uint64_t hp = *hit_pos;
        if (g < uint64_t(d.cap_tuples) && hp + nh <= uint64_t(d.cap_tuple_hits)) {
          d.tuple_off[g] = uint32_t(hp);
          const uint32_t hbase = d.ev[e].hit_base;
          for (int k = 0; k <= depth; ++k) {
            const uint32_t ih = d.cell_inner[stack_c[k]];
            d.tuple_hits[hp + k] = ih;
            d.tuple_det[hp + k] = uint16_t(d.detind[hbase + ih]);
          }
          const uint32_t oh = d.cell_outer[stack_c[depth]];
          d.tuple_hits[hp + depth + 1] = oh;
          d.tuple_det[hp + depth + 1] = uint16_t(d.detind[hbase + oh]);
          d.quality[g] = 0;
          // cell -> track pairs, only for the tuples kept (the event's n_tuples: the
          // reference's cap, or none when the event is past the batch buffers), so that
          // the counts equal the entries k_cell_tracks_fill writes
          if (g - tuple_lo < tcap) {
            const uint64_t pp = hp - g;  // sum over earlier tuples of (hits - 1)
            for (int k = 0; k <= depth; ++k) {
              d.tuple_cell[pp + k] = stack_c[k];
              atomicAdd(&d.ct_cur[stack_c[k]], 1u);
            }
          }
        }
        *tuple_pos = g + 1;
        *hit_pos = hp + nh;
      } else {
        // the tuple's record, appended to the warp's part of the pool
        const uint32_t slot = atomicAdd(&d.tp_ctr[part * kTpStride], 1u);
        if (slot < d.tp_part) {
          const uint64_t r = uint64_t(part) * d.tp_part + slot;
          uint32_t cc[kMaxDepth];
#pragma unroll
          for (int k = 0; k < kMaxDepth; ++k) cc[k] = k <= depth ? stack_c[k] : 0u;
          d.tp_hdr[r] = make_uint4(uint32_t(start), *ntup, *nhit, (uint32_t(e) << 4) | nh);
          d.tp_cells[2 * r] = make_uint4(cc[0], cc[1], cc[2], cc[3]);
          d.tp_cells[2 * r + 1] = make_uint4(cc[4], cc[5], cc[6], cc[7]);
        } else {
          d.tp_ctr[kTpParts * kTpStride] = 1u;  // the fill walks again
        }
        *ntup += 1;
        *nhit += nh;
      }
    }
    --depth;
  }
  (void)cb;
}

__device__ __forceinline__ bool is_start(const Dev& d, uint64_t c) {
  if (d.cell_id[c] < 0) return false;
  const int p = d.cell_pair[c];
  return p < 8 || p > 12;  // minHitsPerNtuplet = 3 (…_impl.jl:125)
}

// Thread per walk: a warp looks at 32 cells at a time and queues in shared memory the
// ones that start a walk (count pass: start cells with at least one neighbour; fill pass:
// start cells the count pass gave tuples), then walks 32 queued cells at once, so that
// every lane of a walking warp has a tree to walk. The count pass writes zero for the
// cells it does not walk; the fill takes each walk's positions from the scanned counts,
// so the order of the walks does not matter.
constexpr int kNtupWarps = 4;
constexpr int kNtupQueue = 64;

template <bool kFill, bool kQ>
__global__ void __launch_bounds__(32 * kNtupWarps) k_ntuplets(Dev d, WorkQueue q) {
  pdl_sync(d);
  __shared__ uint32_t s_queue[kNtupWarps][kNtupQueue];
  // the fill walks only when the count pass could not keep every tuple's record
  if (kFill && d.tp_ctr[kTpParts * kTpStride] == 0) return;
  // The warp's records go to another part after every walk, so that the parts fill alike: with one
  // part per warp, 111 uneven events (40 warps for 70 k tuples of the largest) overflowed some, and the
  // fill walked again (1.93 ms instead of 0.55).
  uint32_t part = ((blockIdx.y * gridDim.x + blockIdx.x) * kNtupWarps + (threadIdx.x >> 5)) % kTpParts;
  for_each_vblock<kQ>(q, [&](int e, uint32_t bx, uint32_t nbx) {
  const EvInfo& E = d.ev[e];
  const uint64_t cb = E.cell_base;
  const unsigned lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
  const unsigned lt = (1u << lane) - 1u;
  const uint32_t ncell = E.n_cells;
  const uint64_t tuple_lo = kFill && ncell > 0 ? d.tstart_cnt[cb] >> 32 : 0;
  // walks the queued cells q0 .. qn (at most 32; lanes past qn idle)
  auto walk_queued = [&](uint32_t q0, uint32_t qn) {
    part = (part + 997u) % kTpParts;
    if (q0 + lane >= qn) return;
    const uint64_t c = cb + s_queue[w][q0 + lane];
    if (!kFill) {
      uint32_t nt = 0, nh = 0;
      walk<false>(d, cb, c, nullptr, nullptr, &nt, &nh, 0, 0, e, part);
      d.tstart_cnt[c] = (uint64_t(nt) << 32) | nh;
    } else {
      const uint64_t v = d.tstart_cnt[c];
      uint64_t tp = v >> 32, hp = v & 0xFFFFFFFFull;
      walk<true>(d, cb, c, &tp, &hp, nullptr, nullptr, tuple_lo, E.n_tuples, e, 0u);
    }
  };
  uint32_t qn = 0;
  for (uint32_t k0 = bx * blockDim.x + 32u * w; k0 < ncell; k0 += nbx * blockDim.x) {
    const uint32_t k = k0 + lane;
    bool walker = false;
    if (k < ncell) {
      const uint64_t c = cb + k;
      if (is_start(d, c)) {
        if (!kFill) walker = d.cn_cnt[c + 1] > d.cn_cnt[c];
        else walker = (d.tstart_cnt[c + 1] >> 32) != (d.tstart_cnt[c] >> 32);
      }
      if (!kFill && !walker) d.tstart_cnt[c] = 0;
    }
    const unsigned b = __ballot_sync(0xffffffffu, walker);
    if (walker) s_queue[w][qn + __popc(b & lt)] = k;
    qn += __popc(b);
    __syncwarp();
    if (qn >= 32) {
      qn -= 32;
      walk_queued(qn, qn + 32);
      __syncwarp();
    }
  }
  walk_queued(0, qn);
  __syncwarp();
  });
}

// The fill from the pool: two blocks per part r move its records to their tuple and hit
// positions (the start cell's scanned positions plus the record's ordinal and hit offset) and
// write what the walking fill writes at a leaf. Independent records, one thread each, so the
// gathers of the tuples' hits overlap; nothing is walked again.
constexpr int kPoolBlocksPerPart = 2;  // measured faster than one (1000 PU50 events: 1.01 / 1.05 ms)

__global__ void __launch_bounds__(256) k_tuples_from_pool(Dev d) {
  pdl_sync(d);
  if (d.tp_ctr[kTpParts * kTpStride]) return;  // a part overflowed: k_ntuplets<true> walks
  for (uint32_t r = blockIdx.x / kPoolBlocksPerPart; r < uint32_t(kTpParts); r += gridDim.x / kPoolBlocksPerPart) {
    uint32_t n = d.tp_ctr[r * kTpStride];
    if (n > d.tp_part) n = d.tp_part;
    for (uint32_t i = threadIdx.x + (blockIdx.x % kPoolBlocksPerPart) * blockDim.x; i < n;
         i += kPoolBlocksPerPart * blockDim.x) {
      const uint64_t s = uint64_t(r) * d.tp_part + i;
      const uint4 h = d.tp_hdr[s];
      const uint4 c0 = d.tp_cells[2 * s], c1 = d.tp_cells[2 * s + 1];
      const uint32_t cells[kMaxDepth] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
      const int e = int(h.w >> 4);
      const uint32_t nh = h.w & 15u;
      const int depth = int(nh) - 2;  // index of the tuple's last doublet
      const uint64_t v = d.tstart_cnt[h.x];
      const uint64_t g = (v >> 32) + h.y;
      const uint64_t hp = (v & 0xFFFFFFFFull) + h.z;
      if (!(g < uint64_t(d.cap_tuples) && hp + nh <= uint64_t(d.cap_tuple_hits))) continue;
      const EvInfo& E = d.ev[e];
      const uint32_t hbase = E.hit_base;
      uint32_t ih[kMaxDepth];
      uint32_t top = 0;
  #pragma unroll
      for (int k = 0; k < kMaxDepth; ++k) {
        ih[k] = k <= depth ? d.cell_inner[cells[k]] : 0u;
        if (k == depth) top = cells[k];
      }
      const uint32_t oh = d.cell_outer[top];
      int16_t det[kMaxDepth];
  #pragma unroll
      for (int k = 0; k < kMaxDepth; ++k)
        if (k <= depth) det[k] = d.detind[hbase + ih[k]];
      const int16_t det_o = d.detind[hbase + oh];
      d.tuple_off[g] = uint32_t(hp);
  #pragma unroll
      for (int k = 0; k < kMaxDepth; ++k)
        if (k <= depth) {
          d.tuple_hits[hp + k] = ih[k];
          d.tuple_det[hp + k] = uint16_t(det[k]);
        }
      d.tuple_hits[hp + depth + 1] = oh;
      d.tuple_det[hp + depth + 1] = uint16_t(det_o);
      d.quality[g] = 0;
      // cell -> track pairs only for the tuples the event keeps (as the walking fill)
      if (g - E.tuple_base < E.n_tuples) {
        const uint64_t pp = hp - g;
  #pragma unroll
        for (int k = 0; k < kMaxDepth; ++k)
          if (k <= depth) {
            d.tuple_cell[pp + k] = cells[k];
            atomicAdd(&d.ct_cur[cells[k]], 1u);
          }
      }
    }
  }
}

__global__ void k_tuple_bases(Dev d) {
  pdl_sync(d);
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e > d.E) return;
  if (e == d.E) {
    const uint64_t v = d.tstart_cnt[d.ev[d.E].n_cells_raw];
    d.ev[e].n_tuples_raw = uint32_t(v >> 32);
    d.ev[e].n_tuple_hits_raw = uint32_t(v);
    d.ev[e].tuple_base = uint32_t(v >> 32);
    d.ev[e].tuple_hit_base = uint32_t(v);
    // the pair list (cell, tuple) holds hits - tuples entries
    return;
  }
  EvInfo& E = d.ev[e];
  const uint64_t lo = d.tstart_cnt[E.cell_base], hi = d.tstart_cnt[uint64_t(E.cell_base) + E.n_cells_raw];
  E.tuple_base = uint32_t(lo >> 32);
  E.tuple_hit_base = uint32_t(lo);
  E.n_tuples_raw = uint32_t(hi >> 32) - uint32_t(lo >> 32);
  E.n_tuple_hits_raw = uint32_t(hi) - uint32_t(lo);
  uint32_t nt = E.n_tuples_raw;
  if (nt > d.tuples_per_event) { nt = d.tuples_per_event; E.warnings |= kWarnTuples; }
  if (uint64_t(E.tuple_base) + E.n_tuples_raw > uint64_t(d.cap_tuples) ||
      uint64_t(E.tuple_hit_base) + E.n_tuple_hits_raw > uint64_t(d.cap_tuple_hits)) {
    E.warnings |= kWarnBuffer;
    nt = 0;
  }
  E.n_tuples = nt;
  for (int b = 0; b < 9; ++b) E.tm_cnt[b] = 0;
  E.tm_done = 0;
}

// Tuple hit offsets end markers and the live sizes for the per-tuple loops. An event with more
// tuples than it keeps ends as the reference's bulk_finalize_fill leaves an overflowing
// container (hist_to_container.jl:150-161): the offset after the last kept tuple is set to that
// tuple's start, so the last kept tuple shows no hits (its doublets still list it).
__global__ void k_tuple_ends(Dev d) {
  pdl_sync(d);
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= d.E) return;
  EvInfo& E = d.ev[e];
  E.n_tuple_hits = 0;
  E.last_tuple_end = 0;
  const uint64_t tb = E.tuple_base;
  if (tb + E.n_tuples_raw <= uint64_t(d.cap_tuples)) {
    d.tuple_off[tb + E.n_tuples_raw] = E.tuple_hit_base + E.n_tuple_hits_raw;
    const uint32_t nt = E.n_tuples;
    if (nt > 0 && nt < E.n_tuples_raw) {
      E.last_tuple_end = d.tuple_off[tb + nt];
      d.tuple_off[tb + nt] = d.tuple_off[tb + nt - 1];
    }
    // hits of the tuples kept (the first n_tuples)
    E.n_tuple_hits = d.tuple_off[tb + nt] - E.tuple_hit_base;
  }
}

// cell -> tuple lists: fill from the (cell, tuple) pairs of the kept tuples
__global__ void k_cell_tracks_fill(Dev d) {
  pdl_sync(d);
  const int e = blockIdx.y;
  // the bitmap that the track lists' sort sets
  for (uint32_t w = (blockIdx.y * gridDim.x + blockIdx.x) * blockDim.x + threadIdx.x, n = d.ev[d.E].n_cells_raw / 32 + 2; w < n;
       w += gridDim.y * gridDim.x * blockDim.x)
    d.dup_bits[w] = 0;
  const EvInfo& E = d.ev[e];
  const uint64_t tb = E.tuple_base;
  for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < E.n_tuples; t += gridDim.x * blockDim.x) {
    const uint64_t g = tb + t;
    // the walk registered every doublet of the last kept tuple, also when its visible size is 0
    const uint32_t h0 = d.tuple_off[g];
    const uint32_t h1 = (t + 1 == E.n_tuples && E.last_tuple_end) ? E.last_tuple_end : d.tuple_off[g + 1];
    const uint64_t pp = uint64_t(h0) - g;
    for (uint32_t k = 0; k + 1 < h1 - h0; ++k) {
      const uint32_t c = d.tuple_cell[pp + k];
      d.ct_list[atomicAdd(&d.ct_cnt[c + 1], 1u)] = uint32_t(g);
    }
  }
}

// kernel_early_duplicate_remover (…_impl.jl:143-166)
template <bool kPerCell>
__global__ void k_early_dup(Dev d) {
  pdl_sync(d);
  const EvInfo& E = d.ev[blockIdx.y];
  for_dup_cells<kPerCell>(d, E, [&](uint32_t k) {
    const uint64_t c = uint64_t(E.cell_base) + k;
    const uint32_t lo = d.ct_cnt[c];
    uint32_t n = d.ct_cnt[c + 1] - lo;
    if (n > uint32_t(kCellRows)) n = kCellRows;
    // kListBatch entries at a time, their loads independent of one another: a cell of 64 tracks
    // otherwise waits for 128 latencies one after the other (42 us for an event of 100 tracks)
    uint32_t maxn = 0;
    for (uint32_t j0 = 0; j0 < n; j0 += kListBatch) {
      uint32_t t[kListBatch], s[kListBatch];
#pragma unroll
      for (int u = 0; u < kListBatch; ++u) t[u] = d.ct_list[lo + min(j0 + u, n - 1)];
#pragma unroll
      for (int u = 0; u < kListBatch; ++u) s[u] = d.tuple_off[t[u] + 1] - d.tuple_off[t[u]];
#pragma unroll
      for (int u = 0; u < kListBatch; ++u) maxn = s[u] > maxn ? s[u] : maxn;
    }
    for (uint32_t j0 = 0; j0 < n; j0 += kListBatch) {
      uint32_t t[kListBatch], s[kListBatch];
#pragma unroll
      for (int u = 0; u < kListBatch; ++u) t[u] = d.ct_list[lo + min(j0 + u, n - 1)];
#pragma unroll
      for (int u = 0; u < kListBatch; ++u) s[u] = d.tuple_off[t[u] + 1] - d.tuple_off[t[u]];
#pragma unroll
      for (int u = 0; u < kListBatch; ++u)
        if (s[u] != maxn) d.quality[t[u]] = 1;
    }
  });
}

// tuple multiplicity counts (kernel_countMultiplicity + finalize!) per event: offsets after
// kernel_fillMultiplicity are the exclusive prefix over bins 1..8. The event's blocks add their
// counts and the last one forms the offsets (one block per event took 180 us for the 51 k tuples of
// an event of pileup 170, most of it on nine shared counters).
__global__ void __launch_bounds__(256) k_multiplicity(Dev d) {
  pdl_sync(d);
  const int e = blockIdx.y;
  EvInfo& E = d.ev[e];
  __shared__ uint32_t s_cnt[9];
  if (threadIdx.x < 9) s_cnt[threadIdx.x] = 0;
  __syncthreads();
  const uint64_t tb = E.tuple_base;
  const uint32_t nt = E.n_tuples;
  uint32_t c[9] = {};  // by hit count, the same in every lane
  for (uint32_t t0 = blockIdx.x * blockDim.x; t0 < nt; t0 += gridDim.x * blockDim.x) {
    const uint32_t t = t0 + threadIdx.x;
    uint32_t n = 0;
    if (t < nt && d.quality[tb + t] != 1) n = d.tuple_off[tb + t + 1] - d.tuple_off[tb + t];
#pragma unroll
    for (uint32_t k = 3; k < 9; ++k) c[k] += __popc(__ballot_sync(0xffffffffu, n == k));
  }
  if ((threadIdx.x & 31u) == 0)
#pragma unroll
    for (int k = 3; k < 9; ++k)
      if (c[k]) atomicAdd(&s_cnt[k - 1], c[k]);
  __syncthreads();
  if (threadIdx.x < 9 && s_cnt[threadIdx.x]) atomicAdd(&E.tm_cnt[threadIdx.x], s_cnt[threadIdx.x]);
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0 && atomicAdd(&E.tm_done, 1u) == gridDim.x - 1) {
    __threadfence();
    uint32_t acc = 0;
    for (int b = 0; b < 9; ++b) {
      const uint32_t n = __ldcg(&E.tm_cnt[b]);
      E.tm_off[b] = acc;
      acc += n;
      if (b >= 2 && b <= 4 && n > d.fits_per_mult) E.warnings |= kWarnFitsCapped;
    }
  }
}

}  // namespace

// CTAs of one persistent wave per tunable stage (SMs x resident CTAs of the stage's
// work-queue kernels, the smaller where a stage has two); 0 for the stages without one
int prepare_ca_kernels(int ctas[kTuneCount]) {
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return -1;
  auto occ = [&](auto kernel, int threads) {
    int n = 0;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, threads, 0) == cudaSuccess ? n : 0;
  };
  for (int s = 0; s < kTuneCount; ++s) ctas[s] = 0;
  ctas[kTuneDoublets] = sms * std::min(occ(k_doublets_count<true>, 256), occ(k_doublets_fill<true>, 256));
  ctas[kTuneConnect] = sms * occ(k_connect_test<true>, 256);
  ctas[kTuneFishbone] = sms * occ(k_fishbone<true>, 128);
  ctas[kTuneNtuplets] = sms * std::min(occ(k_ntuplets<false, true>, 32 * kNtupWarps),
                                       occ(k_ntuplets<true, true>, 32 * kNtupWarps));
  return 0;
}

void launch_ca(const Dev& d, const Launch& L) {
  auto g = [&](int seg) { return dim3(L.bpe_of(seg), d.E); };
  const int eb = div_up(d.E + 1, 128);
  uint32_t* pair_cum = d.pair_cum;
  L.run(k_items, 1 + int(std::min<int64_t>(148, div_up(d.cap_hits, 1024))), 1024, 0, d, pair_cum);
  L.mark("doublet_items");
  // the per-event stages run on their static grid or from a work queue (Launch::queue_of):
  // virtual blocks of (strides x block size) work units, events by decreasing hit count
  if (L.queue_of(kTuneDoublets) || L.queue_of(kTuneConnect) || L.queue_of(kTuneFishbone) || L.queue_of(kTuneNtuplets))
    launch_wq_order(d, L);
  auto plan = [&](int seg, int count_off, int threads) {
    return launch_wq_plan(d, L, count_off, uint32_t(L.queue_of(seg)) * uint32_t(threads));
  };
  const int ctas_dbl = L.queue_of(kTuneDoublets) ? L.wq_ctas[kTuneDoublets] : 0;
  if (ctas_dbl) {
    const WorkQueue q = plan(kTuneDoublets, int(offsetof(EvInfo, n_items)), 256);
    L.run(k_doublets_count<true>, ctas_dbl, 256, 0, d, pair_cum, q);
  } else {
    L.run(k_doublets_count<false>, g(kTuneDoublets), 256, 0, d, pair_cum, WorkQueue{});
  }
  L.mark("doublets_count");
  excl_scan_u32(d.item_cnt, d.cap_items, &d.ev[d.E].n_items, d.scan_tmp, L);
  L.run(k_cell_bases, 1, 1024, 0, d);
  L.mark("doublets_scan");
  if (ctas_dbl) {
    const WorkQueue q = plan(kTuneDoublets, int(offsetof(EvInfo, n_items)), 256);
    L.run(k_doublets_fill<true>, ctas_dbl, 256, 0, d, pair_cum, q);
  } else {
    L.run(k_doublets_fill<false>, g(kTuneDoublets), 256, 0, d, pair_cum, WorkQueue{});
  }
  L.mark("doublets_fill");
  // cells ending on each hit (counted by the doublet fill)
  excl_scan_shift_u32(d.ohc_cur, d.ohc_cnt, d.cap_hits, &d.ev[d.E].n_hits, d.scan_tmp, L);
  L.run(k_ohc_fill, g(kTuneHitLists), 256, 0, d);
  if (d.E <= kPdlEvents) L.run(k_sort_hit_lists, dim3(event_blocks(d.E, 148 * 8, 1024), d.E), 256, 0, d, 4u);
  else L.run(k_sort_hit_lists, g(kTuneHitLists), 256, 0, d, 32u);
  L.mark("outer_hit_lists");
  // connection and neighbour lists
  if (L.queue_of(kTuneConnect)) {
    const WorkQueue q = plan(kTuneConnect, int(offsetof(EvInfo, n_cells)), 256);
    L.run(k_connect_test<true>, L.wq_ctas[kTuneConnect], 256, 0, d, q);
  } else {
    L.run(k_connect_test<false>, g(kTuneConnect), 256, 0, d, WorkQueue{});
  }
  L.mark("connect");
  excl_scan_shift_u32(d.cn_cur, d.cn_cnt, d.cap_cells, &d.ev[d.E].n_cells_raw, d.scan_tmp, L);
  L.run(k_connect_fill, 148 * 8, 256, 0, d);
  L.run(k_sort_cell_lists<0>, g(kTuneCellLists), 256, 0, d);
  L.run(k_sort_long, kSortLongBlocks, 256, 0, d, 0, d.cn_list);
  L.mark("neighbour_lists");
  if (L.queue_of(kTuneFishbone)) {
    const WorkQueue q = plan(kTuneFishbone, int(offsetof(EvInfo, n_hits)), 128);
    L.run(k_fishbone<true>, L.wq_ctas[kTuneFishbone], 128, 0, d, q);
  } else {
    L.run(k_fishbone<false>, g(kTuneFishbone), 128, 0, d, WorkQueue{});
  }
  L.mark("fishbone");
  // ntuplets: the count pass keeps each tuple's record in the pool; the fill moves the records
  // into place, or walks again when the pool overflowed
  const int ctas_nt = L.queue_of(kTuneNtuplets) ? L.wq_ctas[kTuneNtuplets] : 0;
  if (ctas_nt) {
    const WorkQueue q = plan(kTuneNtuplets, int(offsetof(EvInfo, n_cells)), 32 * kNtupWarps);
    L.run(k_ntuplets<false, true>, ctas_nt, 32 * kNtupWarps, 0, d, q);
  } else {
    L.run(k_ntuplets<false, false>, g(kTuneNtuplets), 32 * kNtupWarps, 0, d, WorkQueue{});
  }
  L.mark("ntuplets_count");
  excl_scan_u64(d.tstart_cnt, d.cap_cells, &d.ev[d.E].n_cells_raw, d.scan_tmp64, L);
  L.run(k_tuple_bases, eb, 128, 0, d);
  // all parts advance together in a batch; a few events' records sit in few parts
  L.run(k_tuples_from_pool, d.E <= 16 ? 148 * 8 : kTpParts * kPoolBlocksPerPart, 256, 0, d);
  if (ctas_nt) {
    const WorkQueue q = plan(kTuneNtuplets, int(offsetof(EvInfo, n_cells)), 32 * kNtupWarps);
    L.run(k_ntuplets<true, true>, ctas_nt, 32 * kNtupWarps, 0, d, q);
  } else {
    // the walking fill returns at once unless the pool overflowed: a few blocks per event
    L.run(k_ntuplets<true, false>, dim3(std::min(L.bpe_of(kTuneNtuplets), 8), d.E), 32 * kNtupWarps, 0, d, WorkQueue{});
  }
  L.run(k_tuple_ends, div_up(d.E, 128), 128, 0, d);
  L.mark("ntuplets_fill");
  excl_scan_shift_u32(d.ct_cur, d.ct_cnt, d.cap_cells, &d.ev[d.E].n_cells_raw, d.scan_tmp, L);
  L.run(k_cell_tracks_fill, g(kTuneCellTracks), 256, 0, d);
  L.run(k_sort_cell_lists<1>, g(kTuneCellTracks), 256, 0, d);
  L.run(k_sort_long, kSortLongBlocks, 256, 0, d, 1, d.ct_list);
  L.mark("cell_tracks");
  L.run(d.E <= kPdlEvents ? k_early_dup<true> : k_early_dup<false>, g(kTuneEarlyDup), 256, 0, d);
  L.run(k_multiplicity, dim3(event_blocks(d.E, 148 * 4, 64), d.E), 256, 0, d);
  L.mark("dup_multiplicity");
}

}  // namespace pxl
