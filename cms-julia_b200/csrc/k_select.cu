// Track classification, duplicate cleaning and vertex finding. Restates
// ca_hit_ntuplet_generator_kernels_impl.jl:213-362 (kernel_classify_tracks,
// kernel_fast_duplicate_remover, kernel_count/fill_hit_in_tracks,
// kernel_triplet_cleaner) with the cuts of ca_hit_ntuplet_generator_kernels.jl:79-87,
// and plugin-PixelVertexFinding/gpu_vertex_finder.jl:51-436.
//
// kernel_fast_duplicate_remover is order dependent (a cell sees the marks of the cells before it);
// it is solved as a fixed point over all cells at once. The triplet cleaner only
// ever writes "dup" and tests "!= bad", so its hits run in parallel. Vertex sums keep
// the reference's track order (a warp per vertex hands its tracks' terms over in order).
#include <cstddef>

#include "pxl_internal.cuh"

namespace pxl {

namespace {

constexpr float kChi2Coeff[4] = {0.68177776f, 0.74609577f, -0.08035491f, 0.00315399f};

// kernel_classify_tracks
__global__ void k_classify(Dev d) {
  pdl_sync(d);
  const int e = blockIdx.y;
  EvInfo& E = d.ev[e];
  const uint64_t tb = E.tuple_base;
  if (blockIdx.x == 0 && threadIdx.x == 0) { E.n_dup_cells = 0; E.n_dup_entries = 0; }  // filled by k_dup_cells
  // the hits' tuple counts (k_hit_to_tuple)
  for (uint32_t h = (blockIdx.y * gridDim.x + blockIdx.x) * blockDim.x + threadIdx.x, n = d.ev[d.E].n_hits; h < n;
       h += gridDim.y * gridDim.x * blockDim.x)
    d.htt_cur[h] = 0;
  for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < E.n_tuples; t += gridDim.x * blockDim.x) {
    const uint64_t g = tb + t;
    d.dup_death0[g] = 0xffffffffu;
    d.dup_death1[g] = 0xffffffffu;
    const uint32_t n = d.tuple_off[g + 1] - d.tuple_off[g];
    if (d.quality[g] == 1) continue;
    if (n < 3) continue;
    const float* st = d.t_state + 5 * g;
    bool nan = false;
    for (int k = 0; k < 5; ++k) nan |= isnan(st[k]);
    if (nan) continue;
    const float ptv = d.t_pt[g];
    const float pt = ptv < 10.0f ? ptv : 10.0f;
    const float cut = __fmul_rn(30.0f, __fadd_rn(kChi2Coeff[0], __fmul_rn(pt, __fadd_rn(kChi2Coeff[1],
                      __fmul_rn(pt, __fadd_rn(kChi2Coeff[2], __fmul_rn(pt, kChi2Coeff[3])))))));
    if (__fmul_rn(3.0f, d.t_chi2[g]) >= cut) continue;
    const bool quad = n > 3;
    const float max_tip = quad ? 0.5f : 0.3f, min_pt = quad ? 0.3f : 0.5f, max_zip = 12.0f;
    if (fabsf(st[1]) < max_tip && ptv > min_pt && fabsf(st[4]) < max_zip) d.quality[g] = 2;
  }
}


// kernel_fast_duplicate_remover (…_impl.jl:244-280). The reference walks the cells in order: among
// the loose tracks of a cell the one with the smallest |tip| stays (the first in the list on
// ties) and the others become duplicates, which later cells no longer look at. So a track dies at
// the first cell, in order, that also holds a still-loose track ahead of it in (|tip|, list order).
// Whether that track is still loose there depends only on tracks ahead of it in turn, so the death
// cells are the one fixed point of
//   death(t) = min { c : t in c, a track u ahead of t in c has death(u) >= c },
// reached from "nobody dies" in as many rounds as the longest such chain (three in events of pileup
// 50 and 170). A round takes all cells at once. The walk in order, one warp per event, was a chain
// of shared-memory latencies: 386 us for an event of pileup 50 and 1.92 ms for one of pileup 170.
//
// k_dup_cells gathers the cells with two or more loose tracks (614 of the 4160 cells with two or more
// tracks at pileup 50): the tracks that are not loose can neither stay nor change. The cells carry
// their index, so they are taken in any order.
template <bool kPerCell>
__global__ void __launch_bounds__(256) k_dup_cells(Dev d) {
  pdl_sync(d);
  EvInfo& E = d.ev[blockIdx.y];
  const uint64_t tb = E.tuple_base, c_lo = E.cell_base;
  uint32_t* et = d.dup_et + E.tuple_hit_base;
  uint32_t* ek = d.dup_ek + E.tuple_hit_base;
  for_dup_cells<kPerCell>(d, E, [&](uint32_t k) {
    const uint64_t c = c_lo + k;
    const uint32_t l0 = d.ct_cnt[c];
    uint32_t n = d.ct_cnt[c + 1] - l0;
    if (n > uint32_t(kCellRows)) n = kCellRows;
    uint64_t loose = 0;
    for (uint32_t j0 = 0; j0 < n; j0 += kListBatch) {
      uint32_t t[kListBatch];
#pragma unroll
      for (int u = 0; u < kListBatch; ++u) t[u] = d.ct_list[l0 + min(j0 + u, n - 1)];
      uint32_t m = 0;
#pragma unroll
      for (int u = 0; u < kListBatch; ++u) m |= uint32_t(j0 + u < n && d.quality[t[u]] == 2) << u;
      loose |= uint64_t(m) << j0;
    }
    const uint32_t m = __popcll(loose);
    if (m < 2) return;
    const uint32_t slot = atomicAdd(&E.n_dup_cells, 1u);
    uint32_t o = atomicAdd(&E.n_dup_entries, m);
    d.dup_cell[E.tuple_hit_base / 2 + slot] = k;
    d.dup_rng[E.tuple_hit_base / 2 + slot] = make_uint2(o, m);
    for (; loose; loose &= loose - 1, ++o) {
      const uint32_t t = d.ct_list[l0 + uint32_t(__ffsll(loose) - 1)];
      et[o] = uint32_t(t - tb);
      ek[o] = __float_as_uint(fabsf(d.t_state[5 * size_t(t) + 1]));  // |tip| >= 0 orders as its bits
    }
  });
}
static_assert(kCellRows <= 64, "loose tracks of a cell as a 64-bit mask");

// The rounds, one CTA per event; the death cells (event-local, 0xffffffff: none) start at none
// (k_classify) and sit in global memory, of which an event uses a few KB.
__global__ void k_dup_resolve(Dev d) {
  pdl_sync(d);
  const EvInfo& E = d.ev[blockIdx.x];
  const uint32_t nc = E.n_dup_cells, ne = E.n_dup_entries;
  if (nc == 0) return;
  const uint64_t tb = E.tuple_base;
  const uint32_t* cell = d.dup_cell + E.tuple_hit_base / 2;
  const uint2* rng = d.dup_rng + E.tuple_hit_base / 2;
  const uint32_t* et = d.dup_et + E.tuple_hit_base;
  const uint32_t* ek = d.dup_ek + E.tuple_hit_base;
  uint32_t* cur = d.dup_death0 + tb;
  uint32_t* nxt = d.dup_death1 + tb;
  for (uint32_t round = 0; round <= ne; ++round) {  // every round settles at least one more track
    for (uint32_t i = threadIdx.x; i < nc; i += blockDim.x) {
      const uint32_t c = cell[i];
      const uint2 r = rng[i];
      // nearly all cells have up to four loose tracks: their loads in flight together
      constexpr uint32_t kN = 4;
      uint32_t t[kN], key[kN], best = 0xffffffffu, pos = 0;
      bool alive[kN];
#pragma unroll
      for (uint32_t u = 0; u < kN; ++u) {
        const uint32_t x = r.x + min(u, r.y - 1);
        t[u] = et[x];
        key[u] = ek[x];
      }
#pragma unroll
      for (uint32_t u = 0; u < kN; ++u) alive[u] = u < r.y && __ldcg(&cur[t[u]]) >= c;
#pragma unroll
      for (uint32_t u = 0; u < kN; ++u)
        if (alive[u] && key[u] < best) { best = key[u]; pos = u; }
      for (uint32_t u = kN; u < r.y; ++u) {
        const uint32_t k = ek[r.x + u];
        if (__ldcg(&cur[et[r.x + u]]) >= c && k < best) { best = k; pos = u; }
      }
      if (best == 0xffffffffu) continue;
#pragma unroll
      for (uint32_t u = 0; u < kN; ++u)
        if (u < r.y && (key[u] > best || (key[u] == best && u > pos))) atomicMin(&nxt[t[u]], c);
      for (uint32_t u = kN; u < r.y; ++u) {
        const uint32_t k = ek[r.x + u];
        if (k > best || (k == best && u > pos)) atomicMin(&nxt[et[r.x + u]], c);
      }
    }
    __syncthreads();
    bool moved = false;
    for (uint32_t x = threadIdx.x; x < ne; x += blockDim.x) {
      const uint32_t t = et[x];
      moved |= __ldcg(&cur[t]) != __ldcg(&nxt[t]);
    }
    if (!__syncthreads_or(moved)) break;
    for (uint32_t x = threadIdx.x; x < ne; x += blockDim.x) cur[et[x]] = 0xffffffffu;
    __syncthreads();
    uint32_t* t = cur;
    cur = nxt;
    nxt = t;
  }
  for (uint32_t x = threadIdx.x; x < ne; x += blockDim.x) {
    const uint32_t t = et[x];
    if (__ldcg(&cur[t]) != 0xffffffffu) d.quality[tb + t] = 1;
  }
}

// hit -> loose tuple lists
template <int kPass>
__global__ void k_hit_to_tuple(Dev d) {
  pdl_sync(d);
  const int e = blockIdx.y;
  const EvInfo& E = d.ev[e];
  const uint64_t tb = E.tuple_base;
  const uint32_t hb = E.hit_base;
  for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < E.n_tuples; t += gridDim.x * blockDim.x) {
    const uint64_t g = tb + t;
    if (d.quality[g] != 2) continue;
    const uint32_t h0 = d.tuple_off[g], h1 = d.tuple_off[g + 1];
    for (uint32_t p = h0; p < h1; ++p) {
      const uint32_t h = hb + d.tuple_hits[p];
      if (kPass == 0) atomicAdd(&d.htt_cur[h], 1u);
      else d.htt_list[atomicAdd(&d.htt_cnt[h + 1], 1u)] = uint32_t(g);
    }
  }
}

// kernel_triplet_cleaner over hits; lists ordered by decreasing tuple id as the reference fills them
__global__ void k_triplet_cleaner(Dev d) {
  pdl_sync(d);
  const int e = blockIdx.y;
  const EvInfo& E = d.ev[e];
  const uint32_t hb = E.hit_base;
  for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < E.n_hits; k += gridDim.x * blockDim.x) {
    const uint32_t lo = d.htt_cnt[hb + k], hi = d.htt_cnt[hb + k + 1];
    const uint32_t n = hi - lo;
    uint32_t* L = d.htt_list + lo;
    for (uint32_t p = 1; p < n; ++p) {  // decreasing id
      const uint32_t v = L[p];
      uint32_t q = p;
      while (q > 0 && L[q - 1] < v) { L[q] = L[q - 1]; --q; }
      L[q] = v;
    }
    if (n < 2) continue;
    uint32_t maxnh = 0;
    for (uint32_t j = 0; j < n; ++j) {
      const uint32_t t = L[j];
      const uint32_t s = d.tuple_off[t + 1] - d.tuple_off[t];
      maxnh = s > maxnh ? s : maxnh;
    }
    for (uint32_t j = 0; j < n; ++j) {
      const uint32_t t = L[j];
      if (d.tuple_off[t + 1] - d.tuple_off[t] != maxnh) d.quality[t] = 1;
    }
    if (maxnh > 3) continue;
    float mc = 10000.f;
    uint32_t im = 0xFFFFFFFFu;
    for (uint32_t j = 0; j < n; ++j) {
      const uint32_t t = L[j];
      const float s = fabsf(d.t_state[5 * size_t(t) + 1]);
      if (d.quality[t] != 0 && s < mc) { mc = s; im = t; }
    }
    for (uint32_t j = 0; j < n; ++j) {
      const uint32_t t = L[j];
      if (d.quality[t] != 0 && t != im) d.quality[t] = 1;
    }
  }
}

// ---------------------------------------------------------------- vertices
// One CTA per event. What bounds it is latency: the sums of the fits and of the 2-means splits are
// taken in the reference's track order, so they are serial chains. A warp takes a vertex: its lanes
// read 32 tracks and form their terms (weights, residuals, divisions) at once, and only the
// additions follow one another, handed over by shuffles. With a thread per vertex, each term's
// loads and division sat in the chain too, and an event above the shared-memory capacity (2048
// tracks then) paid global latency for them: an event of pileup 170 (4.3 k tracks) took 5.66 ms
// and one of pileup 50 326 us.
constexpr int kMaxVtx = 1024;
constexpr int kVtxWideThreads = 1024, kVtxNarrowThreads = 256;
// Selected tracks whose arrays fit shared memory. The narrow form (54 KB, four CTAs per SM) serves
// batches that fill the SMs with one CTA per event; the wide form (one CTA per SM) serves small
// batches and the few events above the narrow capacity; above both, global memory.
constexpr uint32_t kVtxWideTracks = 11264, kVtxNarrowTracks = 2048;
constexpr int kVtxParts = 64;  // most blocks that select an event's tracks

struct VtxShared {
  uint32_t sh[33];
  uint32_t off[257];
  uint32_t cur[256];
  uint32_t nv, nvi, warn;
  uint32_t vcnt[kMaxVtx], voff[kMaxVtx + 1];
  int32_t vnd[kMaxVtx];  // the vertices' ndof
  uint16_t parent[kMaxVtx];
};

// per-track arrays of one event, in shared or global memory, by position in z order
template <typename TI, typename TB>
struct VtxTracks {
  float* zt;
  float* ezt2;
  TI* iv;        // 1-based values as the reference stores them; positions until the vertices are numbered
  TI* nn;
  TB* ord;       // the track (in tuple order) at a position
  TB* B;         // the vertices' track lists (positions)
  TB* C;         // scratch
  uint8_t* izt;  // z bins by track; then the 2-means sides by position
};

constexpr size_t vtx_smem_bytes(uint32_t tracks) { return (sizeof(VtxShared) + 15) / 16 * 16 + size_t(tracks) * 19; }

// acc0 + a[0] + a[1] + ... and acc1 + b[0] + ... over the lanes of a warp in lane order (lanes that
// take no part hold +0, which leaves a sum that is never -0 as it is); every lane gets the sums
__device__ __forceinline__ void ordered_add2(float a, float b, uint32_t n, float& acc0, float& acc1) {
  if (n >= 32) {
#pragma unroll
    for (int k = 0; k < 32; ++k) {
      acc0 = __fadd_rn(acc0, __shfl_sync(0xffffffffu, a, k));
      acc1 = __fadd_rn(acc1, __shfl_sync(0xffffffffu, b, k));
    }
  } else {
#pragma unroll 4
    for (uint32_t k = 0; k < n; ++k) {
      acc0 = __fadd_rn(acc0, __shfl_sync(0xffffffffu, a, k));
      acc1 = __fadd_rn(acc1, __shfl_sync(0xffffffffu, b, k));
    }
  }
}

__device__ __forceinline__ float ordered_add(float a, uint32_t n, float acc) {
  if (n >= 32) {
#pragma unroll
    for (int k = 0; k < 32; ++k) acc = __fadd_rn(acc, __shfl_sync(0xffffffffu, a, k));
  } else {
#pragma unroll 4
    for (uint32_t k = 0; k < n; ++k) acc = __fadd_rn(acc, __shfl_sync(0xffffffffu, a, k));
  }
  return acc;
}

// cluster_tracks_by_density, fit_vertices, split_vertices and sort_by_pt2 on the nt selected
// tracks of one event (one CTA); gz, ge, ptt2 and itrk are theirs in tuple order, nn_out receives the
// reference's nn array (neighbour counts of the tracks, then ndof of the vertices).
template <typename TI, typename TB>
__device__ __forceinline__ void vertex_core(Dev& d, EvInfo& E, uint32_t nt, const VtxTracks<TI, TB>& A,
                                            const float* gz, const float* ge, const float* ptt2, const uint32_t* itrk,
                                            float* zv, float* wv, float* vchi2, float* ptv2, uint16_t* sort_ind,
                                            int32_t* nn_out, VtxShared& S) {
  const uint64_t tb = E.tuple_base;
  float* zt = A.zt;
  float* ezt2 = A.ezt2;
  TI* iv = A.iv;
  TI* nn = A.nn;
  TB* ord = A.ord;
  TB* B = A.B;
  TB* C = A.C;
  uint8_t* izt = A.izt;
  const unsigned lane = threadIdx.x & 31u, wid = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  // cluster_tracks_by_density (:84-206), HisToContainer{UInt8,256,16000,8,UInt16}
  for (uint32_t b = threadIdx.x; b < 257; b += blockDim.x) S.off[b] = 0;
  __syncthreads();
  float* z0 = ezt2;  // z in tuple order, until the positions are known
  for (uint32_t i = threadIdx.x; i < nt; i += blockDim.x) {
    const float z = gz[i];
    int32_t iz = int32_t(trunc(__dmul_rn(double(z), 10.)));
    iz = iz < -128 ? -128 : (iz > 127 ? 127 : iz);
    z0[i] = z;
    izt[i] = uint8_t(iz + 128);
    atomicAdd(&S.off[iz + 128], 1u);
  }
  __syncthreads();
  {  // exclusive starts of the 256 bins
    const uint32_t v = threadIdx.x < 256 ? S.off[threadIdx.x] : 0u;
    uint32_t tot;
    const uint32_t ex = block_excl_scan(v, S.sh, &tot);
    if (threadIdx.x < 256) { S.off[threadIdx.x] = ex; S.cur[threadIdx.x] = ex; }
    if (threadIdx.x == 0) S.off[256] = tot;
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < nt; i += blockDim.x) C[atomicAdd(&S.cur[izt[i]], 1u)] = TB(i);
  __syncthreads();
  // Positions in z order (the bins are z ranges; equal z by decreasing track, the reference's order
  // in a bin). The reference scans a track's bin and the two next to it, 1 mm each; in z order the
  // tracks within eps = 0.7 mm are one run around it, which two short walks find: half the pairs,
  // and the arrays read in order (370 k of 600 k cycles of an event of 4.3 k tracks were these scans).
  for (uint32_t i = threadIdx.x; i < nt; i += blockDim.x) {
    const uint32_t b = izt[i], hi = S.off[b + 1];
    const float z = z0[i];
    uint32_t r = S.off[b];
    for (uint32_t q = r; q < hi; ++q) {
      const uint32_t j = C[q];
      const float zj = z0[j];
      r += zj < z || (zj == z && j > i);
    }
    ord[r] = TB(i);
  }
  __syncthreads();
  for (uint32_t s = threadIdx.x; s < nt; s += blockDim.x) zt[s] = z0[ord[s]];
  __syncthreads();
  for (uint32_t s = threadIdx.x; s < nt; s += blockDim.x) ezt2[s] = ge[ord[s]];
  for (uint32_t s = threadIdx.x; s < nt; s += blockDim.x) C[ord[s]] = TB(s);
  __syncthreads();
  const float eps = 0.07f, err2_max = __fmul_rn(0.01f, 0.01f), chi2_max = 9.0f;
  for (uint32_t s = threadIdx.x; s < nt; s += blockDim.x) {
    const float e2 = ezt2[s], z = zt[s];
    int32_t cnt = 0;
    if (!(e2 > err2_max)) {
      auto step = [&](uint32_t p) {
        const float dist = fabsf(__fsub_rn(z, zt[p]));
        if (dist > eps) return false;
        if (!(__fmul_rn(dist, dist) > __fmul_rn(chi2_max, __fadd_rn(e2, ezt2[p])))) ++cnt;
        return true;
      };
      for (uint32_t p = s + 1; p < nt && step(p); ++p) {}
      for (uint32_t p = s; p > 0 && step(p - 1); --p) {}
    }
    nn[s] = TI(cnt);
  }
  __syncthreads();
  // the nearest track of more neighbours (of as many, at smaller z); among equally near ones the
  // last in the reference's order (bins up, tracks down within a bin)
  for (uint32_t s = threadIdx.x; s < nt; s += blockDim.x) {
    const float e2 = ezt2[s], z = zt[s];
    const TI ni = nn[s];
    float mdist = eps;
    uint32_t a = s;
    auto step = [&](uint32_t p) {
      const float zp = zt[p];
      const float dist = fabsf(__fsub_rn(z, zp));
      if (dist > mdist) return false;  // and so are the tracks beyond
      const TI np = nn[p];
      if (np < ni || (np == ni && zp >= z)) return true;
      if (__fmul_rn(dist, dist) > __fmul_rn(chi2_max, __fadd_rn(e2, ezt2[p]))) return true;
      if (dist == mdist && a != s) {
        const uint32_t ip = ord[p], ia = ord[a];
        const uint8_t bp = izt[ip], ba = izt[ia];
        if (bp != ba ? bp < ba : ip > ia) return true;
      }
      mdist = dist;
      a = p;
      return true;
    };
    for (uint32_t p = s + 1; p < nt && step(p); ++p) {}
    for (uint32_t p = s; p > 0 && step(p - 1); --p) {}
    iv[s] = TI(a + 1);
  }
  __syncthreads();
  for (uint32_t s = threadIdx.x; s < nt; s += blockDim.x) {
    int32_t m = iv[s];
    while (m != int32_t(iv[m - 1])) m = iv[m - 1];
    iv[s] = TI(m);
  }
  __syncthreads();
  uint32_t found = 0;  // vertices are numbered in tuple order
  for (uint32_t b = 0; b < nt; b += blockDim.x) {
    const uint32_t i = b + threadIdx.x;
    const uint32_t s = i < nt ? C[i] : 0u;
    const bool root = i < nt && iv[s] == TI(s + 1);
    const bool seed = root && nn[s] >= 2;
    uint32_t tot;
    const uint32_t ex = block_excl_scan(seed ? 1u : 0u, S.sh, &tot);
    if (root) iv[s] = TI(seed ? -int32_t(found + ex + 1) : -9998);
    found += tot;
  }
  __syncthreads();
  for (uint32_t s = threadIdx.x; s < nt; s += blockDim.x)
    if (iv[s] >= 0) iv[s] = iv[iv[s] - 1];
  __syncthreads();
  for (uint32_t s = threadIdx.x; s < nt; s += blockDim.x) iv[s] = TI(-iv[s]);
  if (threadIdx.x == 0) {
    if (found >= uint32_t(kMaxVtx)) { S.warn |= kWarnVertex; found = kMaxVtx - 1; }
    S.nv = found;
    S.nvi = found;
  }
  __syncthreads();
  // per-vertex track lists in ascending track order (the order of the reference's loops over
  // all tracks). A vertex made by a split keeps its parent's
  // list and selects its own tracks by id, as the loops over all tracks do.
  const uint32_t nv0 = S.nv;
  for (uint32_t v = threadIdx.x; v < uint32_t(kMaxVtx); v += blockDim.x) { S.vcnt[v] = 0; S.parent[v] = uint16_t(v); }
  __syncthreads();
  for (uint32_t s = threadIdx.x; s < nt; s += blockDim.x)
    if (iv[s] >= 1 && uint32_t(iv[s]) <= nv0) atomicAdd(&S.vcnt[iv[s] - 1], 1u);
  __syncthreads();
  {
    uint32_t base = 0;
    for (uint32_t b = 0; b < nv0; b += blockDim.x) {
      const uint32_t v = b + threadIdx.x;
      const uint32_t c = v < nv0 ? S.vcnt[v] : 0u;
      uint32_t tot;
      const uint32_t ex = block_excl_scan(c, S.sh, &tot);
      if (v < nv0) { S.voff[v] = base + ex; S.vcnt[v] = base + ex; }
      base += tot;
    }
    if (threadIdx.x == 0) S.voff[nv0] = base;
  }
  __syncthreads();
  for (uint32_t s = threadIdx.x; s < nt; s += blockDim.x)
    if (iv[s] >= 1 && uint32_t(iv[s]) <= nv0) C[atomicAdd(&S.vcnt[iv[s] - 1], 1u)] = ord[s];
  __syncthreads();
  for (uint32_t s = threadIdx.x; s < nt; s += blockDim.x)
    if (iv[s] >= 1 && uint32_t(iv[s]) <= nv0) {  // its rank among the vertex's tracks
      const TB i = ord[s];
      uint32_t r = S.voff[iv[s] - 1];
      for (uint32_t q = r, hi = S.voff[iv[s]]; q < hi; ++q) r += C[q] < i;
      B[r] = TB(s);
    }
  __syncthreads();
  // fit_vertices, :228-286: a warp per vertex, its sums in track order
  auto fit = [&](double chi2max) {
    const uint32_t nvf = S.nvi;
    for (uint32_t v = wid; v < nvf; v += nwarp) {
      const uint32_t pv = S.parent[v], lo = S.voff[pv], hi = S.voff[pv + 1];
      float z = 0, w = 0;
      for (uint32_t p0 = lo; p0 < hi; p0 += 32) {
        float wi = 0.f, zw = 0.f;
        if (p0 + lane < hi) {
          const uint32_t i = B[p0 + lane];
          if (iv[i] == int32_t(v + 1)) {
            wi = __fdiv_rn(1.0f, ezt2[i]);
            zw = __fmul_rn(zt[i], wi);
          }
        }
        ordered_add2(zw, wi, hi - p0, z, w);
      }
      if (!(w > 0) && lane == 0) atomicOr(&S.warn, kWarnVertex);
      z = __fdiv_rn(z, w);
      float c2s = 0;
      int32_t cnt = -1;
      for (uint32_t p0 = lo; p0 < hi; p0 += 32) {
        float c2 = 0.f;
        bool in = false;
        if (p0 + lane < hi) {
          const uint32_t i = B[p0 + lane];
          if (iv[i] == int32_t(v + 1)) {
            c2 = __fsub_rn(z, zt[i]);
            c2 = __fmul_rn(c2, __fdiv_rn(c2, ezt2[i]));
            in = !(double(c2) > chi2max);
            if (!in) { iv[i] = 9999; c2 = 0.f; }
          }
        }
        cnt += __popc(__ballot_sync(0xffffffffu, in));
        c2s = ordered_add(c2, hi - p0, c2s);
      }
      if (cnt > 0) w = __fmul_rn(w, __fdiv_rn(float(cnt), c2s));
      if (lane == 0) { zv[v] = z; wv[v] = w; vchi2[v] = c2s; S.vnd[v] = cnt; }
    }
    __syncthreads();
    if (threadIdx.x == 0) S.nv = nvf;
    __syncthreads();
  };
  fit(50.);
  // split_vertices, :288-371: each vertex decides alone; new ids follow the vertex order
  {
    const uint32_t nvf = S.nv;
    for (uint32_t kv = wid; kv < nvf; kv += nwarp) {
      bool split = false;
      const uint32_t lo = S.voff[kv], hi = S.voff[kv + 1];
      if (S.vnd[kv] >= 4 && !(vchi2[kv] < __fmul_rn(9.0f, float(S.vnd[kv])))) {
        if (S.vnd[kv] >= 512) {
          if (lane == 0) atomicOr(&S.warn, kWarnVertex);
        } else {
          // 2-means in the vertex's tracks (zz = zt - zv, weights 1/ezt2), at most 20 iterations;
          // first assignment: zz < 0 -> 1 else 2, kept per track in izt
          uint32_t nq = 0;
          const float zc = zv[kv];
          for (uint32_t p0 = lo; p0 < hi; p0 += 32) {
            bool in = false;
            if (p0 + lane < hi) {
              const uint32_t i = B[p0 + lane];
              in = iv[i] == int32_t(kv + 1);
              if (in) izt[i] = __fsub_rn(zt[i], zc) < 0 ? 1 : 2;
            }
            nq += __popc(__ballot_sync(0xffffffffu, in));
          }
          if (nq != uint32_t(S.vnd[kv] + 1) && lane == 0) atomicOr(&S.warn, kWarnVertex);
          bool more = true;
          int iter = 20;
          float znew0 = 0, znew1 = 0, w0 = 0, w1 = 0;
          while (more) {
            znew0 = znew1 = 0; w0 = w1 = 0;
            for (uint32_t p0 = lo; p0 < hi; p0 += 32) {
              float ww = 0.f, zw = 0.f;
              bool first = false;
              if (p0 + lane < hi) {
                const uint32_t i = B[p0 + lane];
                if (iv[i] == int32_t(kv + 1)) {
                  ww = __fdiv_rn(1.0f, ezt2[i]);
                  zw = __fmul_rn(__fsub_rn(zt[i], zc), ww);
                  first = izt[i] == 1;
                }
              }
              const uint32_t m1 = __ballot_sync(0xffffffffu, first);
              const uint32_t n = hi - p0 < 32 ? hi - p0 : 32;
#pragma unroll 4
              for (uint32_t k = 0; k < n; ++k) {
                const float a = __shfl_sync(0xffffffffu, zw, k), b = __shfl_sync(0xffffffffu, ww, k);
                if ((m1 >> k) & 1u) { znew0 = __fadd_rn(znew0, a); w0 = __fadd_rn(w0, b); }
                else { znew1 = __fadd_rn(znew1, a); w1 = __fadd_rn(w1, b); }
              }
            }
            znew0 = __fdiv_rn(znew0, w0);
            znew1 = __fdiv_rn(znew1, w1);
            bool moved = false;
            for (uint32_t p = lo + lane; p < hi; p += 32) {
              const uint32_t i = B[p];
              if (iv[i] != int32_t(kv + 1)) continue;
              const float zz = __fsub_rn(zt[i], zc);
              const float d0 = fabsf(__fsub_rn(znew0, zz)), d1 = fabsf(__fsub_rn(znew1, zz));
              const uint8_t newer = d0 < d1 ? 1 : 2;
              moved |= newer != izt[i];
              izt[i] = newer;
            }
            more = __any_sync(0xffffffffu, moved);
            if (--iter <= 0) more = false;
          }
          if (!(w0 == 0 || w1 == 0)) {
            const float dd = __fsub_rn(znew0, znew1);
            const float dist2 = __fmul_rn(dd, dd);
            const float chi2_dist = __fdiv_rn(dist2, __fadd_rn(__fdiv_rn(1.0f, w0), __fdiv_rn(1.0f, w1)));
            split = !(chi2_dist < 4);
          }
        }
      }
      if (lane == 0) S.vcnt[kv] = split ? 1u : 0u;
    }
    __syncthreads();
    // ids of the new vertices (0xffffffff: not split)
    uint32_t base = S.nvi;
    for (uint32_t b = 0; b < nvf; b += blockDim.x) {
      const uint32_t kv = b + threadIdx.x;
      const bool split = kv < nvf && S.vcnt[kv] != 0;
      uint32_t tot;
      const uint32_t slot = base + block_excl_scan(split ? 1u : 0u, S.sh, &tot);
      if (split && slot < uint32_t(kMaxVtx)) S.parent[slot] = uint16_t(kv);
      if (kv < nvf) S.vcnt[kv] = split ? slot : 0xffffffffu;
      base += tot;
    }
    __syncthreads();
    for (uint32_t kv = wid; kv < nvf; kv += nwarp) {
      const uint32_t slot = S.vcnt[kv];
      if (slot == 0xffffffffu) continue;
      for (uint32_t p = S.voff[kv] + lane; p < S.voff[kv + 1]; p += 32) {
        const uint32_t i = B[p];
        if (iv[i] == int32_t(kv + 1) && izt[i] == 2) iv[i] = TI(slot + 1);
      }
    }
    if (threadIdx.x == 0) {
      if (base >= uint32_t(kMaxVtx)) { atomicOr(&S.warn, kWarnVertex); base = kMaxVtx - 1; }
      S.nvi = base;
    }
    __syncthreads();
  }
  fit(5000.);
  // sort_by_pt2, :391-436 (the sorted order itself is dropped by the reference)
  const uint32_t nvf = S.nv;
  if (nvf >= 1) {
    for (uint32_t s = threadIdx.x; s < nt; s += blockDim.x) d.idv[tb + itrk[ord[s]]] = int16_t(iv[s]);
    for (uint32_t v = wid; v < nvf; v += nwarp) {
      const uint32_t pv = S.parent[v], lo = S.voff[pv], hi = S.voff[pv + 1];
      float s = 0;
      for (uint32_t p0 = lo; p0 < hi; p0 += 32) {
        float x = 0.f;
        if (p0 + lane < hi) {
          const uint32_t i = B[p0 + lane];
          if (iv[i] == int32_t(v + 1)) x = ptt2[ord[i]];
        }
        s = ordered_add(x, hi - p0, s);
      }
      if (lane == 0) ptv2[v] = s;
    }
    if (threadIdx.x == 0 && nvf == 1) sort_ind[0] = 1;
  }
  for (uint32_t s = threadIdx.x; s < nt; s += blockDim.x)
    if (ord[s] >= nvf) nn_out[ord[s]] = nn[s];
  for (uint32_t v = threadIdx.x; v < nvf; v += blockDim.x) nn_out[v] = S.vnd[v];
  __syncthreads();
  if (threadIdx.x == 0) {
    E.n_vtx = nvf;
    if (S.warn) E.warnings |= S.warn;
  }
}

// load_tracks (:51-82): the event's tracks of >= 4 hits, loose, pt >= 0.5, in tuple order. Each of
// the event's blocks lists those of its range of tuples (vws_list, vtx_cnt); it also clears the range's
// vertex ids and, with the first block, the event's vertex products.
__global__ void __launch_bounds__(256) k_vertex_select(Dev d) {
  pdl_sync(d);
  const int e = blockIdx.y;
  const EvInfo& E = d.ev[e];
  __shared__ uint32_t sh[33];
  if (blockIdx.x == 0)
    for (uint32_t v = threadIdx.x; v < uint32_t(kMaxVtx); v += blockDim.x) {
      const size_t g = size_t(e) * kMaxVtx + v;
      d.zv[g] = 0; d.wv[g] = 0; d.vchi2[g] = 0; d.ptv2[g] = 0; d.sort_ind[g] = 0;
    }
  const uint64_t tb = E.tuple_base;
  const uint32_t per = (E.n_tuples + gridDim.x - 1) / gridDim.x;
  const uint32_t lo = min(E.n_tuples, blockIdx.x * per), hi = min(E.n_tuples, lo + per);
  uint32_t n = 0;
  for (uint32_t b = lo; b < hi; b += blockDim.x) {
    const uint32_t t = b + threadIdx.x;
    bool sel = false;
    if (t < hi) {
      d.idv[tb + t] = -1;
      sel = d.tuple_off[tb + t + 1] - d.tuple_off[tb + t] >= 4 && d.quality[tb + t] == 2 && !(d.t_pt[tb + t] < 0.5f);
    }
    uint32_t tot;
    const uint32_t r = n + block_excl_scan(sel ? 1u : 0u, sh, &tot);
    if (sel) d.vws_list[tb + lo + r] = t;
    n += tot;
  }
  if (threadIdx.x == 0) d.vtx_cnt[e * gridDim.x + blockIdx.x] = n;
}

// Events of the grid's stride with more than `above` selected tracks, and at most kCap (kAll: those
// above too, in global memory). parts: blocks of k_vertex_select per event.
template <int kThreads, uint32_t kCap, bool kAll>
__global__ void __launch_bounds__(kThreads, kAll ? 1 : 4) k_vertices(Dev d, int parts, uint32_t above) {
  pdl_sync(d);
  extern __shared__ __align__(16) uint8_t s_vtx[];
  VtxShared& S = *reinterpret_cast<VtxShared*>(s_vtx);
  float* s_zt = reinterpret_cast<float*>(s_vtx + (sizeof(VtxShared) + 15) / 16 * 16);
  float* s_ezt2 = s_zt + kCap;
  int16_t* s_iv = reinterpret_cast<int16_t*>(s_ezt2 + kCap);
  int16_t* s_nn = s_iv + kCap;
  uint16_t* s_ord = reinterpret_cast<uint16_t*>(s_nn + kCap);
  uint16_t* s_b = s_ord + kCap;
  uint16_t* s_c = s_b + kCap;
  uint8_t* s_izt = reinterpret_cast<uint8_t*>(s_c + kCap);
  for (int e = blockIdx.x; e < d.E; e += gridDim.x) {
    EvInfo& E = d.ev[e];
    const uint64_t tb = E.tuple_base;
    // the blocks' lists, one after the other
    uint32_t nt;
    const uint32_t c = threadIdx.x < uint32_t(parts) ? d.vtx_cnt[e * parts + threadIdx.x] : 0u;
    const uint32_t first = block_excl_scan(c, S.sh, &nt);
    if (threadIdx.x < uint32_t(parts)) S.off[threadIdx.x] = first;
    __syncthreads();
    if (nt <= above && above > 0) continue;
    if (!kAll && nt > kCap) continue;
    const uint32_t per = (E.n_tuples + parts - 1) / parts;
    for (uint32_t i = threadIdx.x; i < nt; i += blockDim.x) {
      uint32_t a = 0, b = uint32_t(parts);
      while (b - a > 1) {
        const uint32_t m = (a + b) >> 1;
        if (S.off[m] <= i) a = m; else b = m;
      }
      const uint32_t t = d.vws_list[tb + a * per + (i - S.off[a])];
      const uint64_t g = tb + t;
      const float pt = d.t_pt[g];
      d.vws_itrk[tb + i] = t;
      d.vws_zt[tb + i] = d.t_state[5 * g + 4];
      d.vws_ezt2[tb + i] = d.t_cov[15 * g + 14];
      d.vws_ptt2[tb + i] = __fmul_rn(pt, pt);
    }
    if (threadIdx.x == 0) { E.n_vtx_tracks = nt; S.warn = 0; }
    __syncthreads();
    float* zv = d.zv + size_t(e) * kMaxVtx;
    float* wv = d.wv + size_t(e) * kMaxVtx;
    float* vchi2 = d.vchi2 + size_t(e) * kMaxVtx;
    float* ptv2 = d.ptv2 + size_t(e) * kMaxVtx;
    uint16_t* sort_ind = d.sort_ind + size_t(e) * kMaxVtx;
    int32_t* nn_out = d.ndof + tb + size_t(e) * kMaxVtx;  // length n_tuples + 1024
    const float* gz = d.vws_zt + tb;
    const float* ge = d.vws_ezt2 + tb;
    const float* ptt2 = d.vws_ptt2 + tb;
    const uint32_t* itrk = d.vws_itrk + tb;
    if (nt <= kCap) {
      const VtxTracks<int16_t, uint16_t> A{s_zt, s_ezt2, s_iv, s_nn, s_ord, s_b, s_c, s_izt};
      vertex_core(d, E, nt, A, gz, ge, ptt2, itrk, zv, wv, vchi2, ptv2, sort_ind, nn_out, S);
    } else if (kAll) {
      const VtxTracks<int32_t, uint32_t> A{d.vws_zs + tb, d.vws_es + tb, d.vws_iv + tb, d.vws_nn + tb,
                                           d.vws_ord + tb, d.vws_bins + tb, d.vws_list + tb, d.vws_izt + tb};
      vertex_core(d, E, nt, A, gz, ge, ptt2, itrk, zv, wv, vchi2, ptv2, sort_ind, nn_out, S);
    }
    __syncthreads();
  }
}

}  // namespace

void launch_classify(const Dev& d, const Launch& L) {
  auto g = [&](int seg) { return dim3(L.bpe_of(seg), d.E); };
  L.run(k_classify, g(kTuneClassify), 256, 0, d);
  L.mark("classify");
  L.run(d.E <= kPdlEvents ? k_dup_cells<true> : k_dup_cells<false>, g(kTuneClassify), 256, 0, d);
  // a CTA per event: many threads where an SM has one event to itself, several events per SM else
  L.run(k_dup_resolve, d.E, d.E <= 148 ? 1024 : 256, 0, d);
  L.mark("fast_duplicate_remover");
  L.run(k_hit_to_tuple<0>, g(kTuneHitToTuple), 256, 0, d);
  excl_scan_shift_u32(d.htt_cur, d.htt_cnt, d.cap_hits, &d.ev[d.E].n_hits, d.scan_tmp, L);
  L.run(k_hit_to_tuple<1>, g(kTuneHitToTuple), 256, 0, d);
  L.mark("hit_to_tuple");
  L.run(k_triplet_cleaner, g(kTuneHitToTuple), 256, 0, d);
  L.mark("triplet_cleaner");
}

int prepare_select_kernels() {
  const int wide = int(vtx_smem_bytes(kVtxWideTracks)), narrow = int(vtx_smem_bytes(kVtxNarrowTracks));
  cudaError_t err = cudaFuncSetAttribute(k_vertices<kVtxWideThreads, kVtxWideTracks, true>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, wide);
  if (err == cudaSuccess)
    err = cudaFuncSetAttribute(k_vertices<kVtxNarrowThreads, kVtxNarrowTracks, false>,
                               cudaFuncAttributeMaxDynamicSharedMemorySize, narrow);
  return err == cudaSuccess ? 0 : -1;
}

void launch_vertices(const Dev& d, const Launch& L) {
  const size_t wide = vtx_smem_bytes(kVtxWideTracks), narrow = vtx_smem_bytes(kVtxNarrowTracks);
  const int parts = event_blocks(d.E, kVtxSelectBlocks, kVtxParts);
  L.run(k_vertex_select, dim3(parts, d.E), 256, 0, d);
  if (d.E <= 148) {  // at most one event per SM: the wide form for all
    L.run(k_vertices<kVtxWideThreads, kVtxWideTracks, true>, d.E, kVtxWideThreads, wide, d, parts, 0u);
  } else {
    L.run(k_vertices<kVtxNarrowThreads, kVtxNarrowTracks, false>, d.E, kVtxNarrowThreads, narrow, d, parts, 0u);
    if (d.tuples_per_event > kVtxNarrowTracks)
      L.run(k_vertices<kVtxWideThreads, kVtxWideTracks, true>, 148, kVtxWideThreads, wide, d, parts, kVtxNarrowTracks);
  }
  L.mark("vertices");
}

}  // namespace pxl
