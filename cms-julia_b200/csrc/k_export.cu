// Batched, stream-ordered copy-out of the track and vertex collections (pxl_export_async).
//
// The reference hands each event's TrackSOA (CUDADataFormats/PixelTrackHeterogeneous.jl:10-62)
// and ZVertexSoA (z_vertex_soa.jl:4-26) to its consumers. For a batch, copying every event's
// fixed-stride views one by one costs one synchronous copy per product per event. Here the
// tracks of quality loose (the ones the vertex finder and downstream consumers take) and the
// vertices of all events are compacted on the device, event after event in tuple order, into
// one packed array per field, and each array goes to host memory in ONE asynchronous copy on
// a copy stream, with no host synchronisation. Two export buffer sets alternate, so the copy of
// one batch overlaps the chain of the next.
#include <algorithm>
#include <cstdio>

#include "../../include/pxl.h"
#include "pxl_ctx.h"
#include "pxl_internal.cuh"

namespace pxl {

namespace {

constexpr int kExpThreads = 256;

// An event's tuples are cut into gridDim.x equal ranges, one per block (event_blocks: one block took
// 1.04 ms to fill the tracks of an event of 51 k tuples, mostly waiting on its scans).
__device__ __forceinline__ uint2 export_range(uint32_t n) {
  const uint32_t per = (n + gridDim.x - 1) / gridDim.x;
  const uint32_t lo = min(n, blockIdx.x * per);
  return make_uint2(lo, min(n, lo + per));
}

// loose tracks per block, vertices per event
__global__ void __launch_bounds__(kExpThreads) k_export_count(Dev d, ExportSet x) {
  pdl_sync(d);
  const int e = blockIdx.y;
  const EvInfo& E = d.ev[e];
  const uint2 r = export_range(E.n_tuples);
  uint32_t tot = 0;
  for (uint32_t b = r.x; b < r.y; b += kExpThreads) {
    const uint32_t t = b + threadIdx.x;
    tot += __syncthreads_count(t < r.y && d.quality[uint64_t(E.tuple_base) + t] == 2);
  }
  if (threadIdx.x == 0) {
    x.block[e * gridDim.x + blockIdx.x] = tot;
    if (blockIdx.x == 0) x.index[4 * e + 3] = E.n_vtx;
  }
}

// first track of each block, first track and first vertex of each event (one block); row E holds
// the totals
__global__ void __launch_bounds__(1024) k_export_scan(Dev d, ExportSet x, int nb) {
  pdl_sync(d);
  __shared__ uint32_t sh[33];
  uint32_t ct = 0, cv = 0;
  for (int b = 0; b < d.E * nb; b += blockDim.x) {
    const int i = b + threadIdx.x;
    uint32_t tot;
    const uint32_t first = ct + block_excl_scan(i < d.E * nb ? x.block[i] : 0u, sh, &tot);
    if (i < d.E * nb) {
      x.block[i] = first;
      if (i % nb == 0) x.index[4 * (i / nb)] = first;
    }
    ct += tot;
  }
  for (int b = 0; b < d.E; b += blockDim.x) {
    const int e = b + threadIdx.x;
    uint32_t tot;
    const uint32_t first = cv + block_excl_scan(e < d.E ? x.index[4 * e + 3] : 0u, sh, &tot);
    if (e < d.E) x.index[4 * e + 2] = first;
    cv += tot;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < d.E; e += blockDim.x)
    x.index[4 * e + 1] = (e + 1 < d.E ? x.index[4 * (e + 1)] : ct) - x.index[4 * e];
  if (threadIdx.x == 0) {
    x.index[4 * d.E] = ct; x.index[4 * d.E + 1] = ct; x.index[4 * d.E + 2] = cv; x.index[4 * d.E + 3] = cv;
  }
}

// the event's loose tracks in tuple order, and its vertices. The tracks of 256 tuples are listed
// in shared memory and their rows copied word by word, so that the stores coalesce.
__global__ void __launch_bounds__(kExpThreads) k_export_fill(Dev d, ExportSet x) {
  pdl_sync(d);
  const int e = blockIdx.y;
  const EvInfo& E = d.ev[e];
  __shared__ uint32_t sh[33];
  __shared__ uint32_t s_src[kExpThreads];
  const uint64_t tb = E.tuple_base;
  const uint2 range = export_range(E.n_tuples);
  uint32_t base = x.block[e * gridDim.x + blockIdx.x];
  for (uint32_t b = range.x; b < range.y; b += kExpThreads) {
    const uint32_t t = b + threadIdx.x;
    const bool loose = t < range.y && d.quality[tb + t] == 2;
    uint32_t tot;
    const uint32_t r = block_excl_scan(loose ? 1u : 0u, sh, &tot);
    if (loose) s_src[r] = t;
    __syncthreads();
    const uint32_t m = base < x.cap_tracks ? min(tot, x.cap_tracks - base) : 0u;
    for (uint32_t w = threadIdx.x; w < 5 * m; w += kExpThreads)
      x.state[5 * size_t(base) + w] = d.t_state[5 * (tb + s_src[w / 5]) + w % 5];
    for (uint32_t w = threadIdx.x; w < 15 * m; w += kExpThreads)
      x.cov[15 * size_t(base) + w] = d.t_cov[15 * (tb + s_src[w / 15]) + w % 15];
    if (threadIdx.x < m) {
      const uint32_t ti = s_src[threadIdx.x];
      const uint64_t g = tb + ti;
      const size_t o = size_t(base) + threadIdx.x;
      x.pt[o] = d.t_pt[g];
      x.eta[o] = d.t_eta[g];
      x.chi2[o] = d.t_chi2[g];
      x.n_hits[o] = uint8_t(d.tuple_off[g + 1] - d.tuple_off[g]);
      x.vertex[o] = d.idv[g];
      x.tuple[o] = ti + 1;
    }
    base += tot;
    __syncthreads();
  }
  if (blockIdx.x != 0) return;
  const uint32_t v0 = x.index[4 * e + 2], nv = E.n_vtx;
  const int32_t* nn = d.ndof + tb + size_t(e) * 1024;
  for (uint32_t v = threadIdx.x; v < nv; v += blockDim.x) {
    const uint32_t o = v0 + v;
    if (o >= x.cap_vertices) break;
    x.zv[o] = d.zv[size_t(e) * 1024 + v];
    x.wv[o] = d.wv[size_t(e) * 1024 + v];
    x.vchi2[o] = d.vchi2[size_t(e) * 1024 + v];
    x.ptv2[o] = d.ptv2[size_t(e) * 1024 + v];
    x.ndof[o] = nn[v];
  }
}

constexpr int kExpBlocks = 148 * 16;  // blocks of the export's kernels (event_blocks); 148 * 4 left 111 uneven
                                       // events five each: their export 1110 us, now 898; 148 * 32: 886

// The packed arrays to host memory that the device can write (pinned), the rows there are and no more.
// For small batches, in place of a copy of each array's whole capacity: 14 copies of 3.2 MB in all take
// 100 us for the 145 KB of tracks of one event of pileup 50 (its chain and export: 684 us, now 588;
// an event of 100 tracks: 461, now 366; the export of eight events of pileup 200, 4.6 MB, 1056, now 136).
// Larger batches keep the copy engine, which leaves the SMs to the next chain.
__device__ __forceinline__ void copy_rows(void* dst, const void* src, size_t bytes) {
  if (!dst) return;
  const size_t first = blockIdx.x * size_t(blockDim.x) + threadIdx.x, stride = size_t(gridDim.x) * blockDim.x;
  for (size_t i = first; i < bytes / 4; i += stride) static_cast<uint32_t*>(dst)[i] = static_cast<const uint32_t*>(src)[i];
  for (size_t i = bytes / 4 * 4 + first; i < bytes; i += stride) static_cast<uint8_t*>(dst)[i] = static_cast<const uint8_t*>(src)[i];
}

constexpr int kExpOutBlocks = 32;

__global__ void __launch_bounds__(kExpThreads) k_export_out(ExportSet x, PxlExport out, int E) {
  pdl_sync();
  const size_t mt = min(size_t(x.index[4 * E + 1]), min(size_t(out.max_tracks), size_t(x.cap_tracks)));
  const size_t mv = min(size_t(x.index[4 * E + 3]), min(size_t(out.max_vertices), size_t(x.cap_vertices)));
  copy_rows(out.index, x.index, size_t(E + 1) * 16);
  copy_rows(out.state, x.state, mt * 20);
  copy_rows(out.cov, x.cov, mt * 60);
  copy_rows(out.pt, x.pt, mt * 4);
  copy_rows(out.eta, x.eta, mt * 4);
  copy_rows(out.chi2, x.chi2, mt * 4);
  copy_rows(out.n_hits, x.n_hits, mt);
  copy_rows(out.vertex, x.vertex, mt * 2);
  copy_rows(out.tuple, x.tuple, mt * 4);
  copy_rows(out.zv, x.zv, mv * 4);
  copy_rows(out.wv, x.wv, mv * 4);
  copy_rows(out.vchi2, x.vchi2, mv * 4);
  copy_rows(out.ptv2, x.ptv2, mv * 4);
  copy_rows(out.ndof, x.ndof, mv * 4);
}

// whether the device can write all of each array of `out` (pinned from its first byte to its last), on
// the word boundaries that copy_rows takes
bool device_writable(const PxlExport& out, int E) {
  const size_t mt = size_t(out.max_tracks), mv = size_t(out.max_vertices);
  const struct {
    const void* p;
    size_t bytes;
  } arrays[] = {{out.index, size_t(E + 1) * 16}, {out.state, mt * 20}, {out.cov, mt * 60}, {out.pt, mt * 4},
                {out.eta, mt * 4}, {out.chi2, mt * 4}, {out.n_hits, mt}, {out.vertex, mt * 2}, {out.tuple, mt * 4},
                {out.zv, mv * 4}, {out.wv, mv * 4}, {out.vchi2, mv * 4}, {out.ptv2, mv * 4}, {out.ndof, mv * 4}};
  for (const auto& a : arrays) {
    if (!a.p || a.bytes == 0) continue;
    if (reinterpret_cast<uintptr_t>(a.p) % 4 != 0) return false;
    for (const char* q : {static_cast<const char*>(a.p), static_cast<const char*>(a.p) + a.bytes - 1}) {
      cudaPointerAttributes t{};
      if (cudaPointerGetAttributes(&t, q) != cudaSuccess) {
        cudaGetLastError();
        return false;
      }
      if (t.type != cudaMemoryTypeHost || t.devicePointer != q) return false;
    }
  }
  return true;
}

template <class T>
cudaError_t alloc_n(T** p, size_t n) {
  return cudaMalloc(reinterpret_cast<void**>(p), std::max<size_t>(n, 1) * sizeof(T));
}

}  // namespace

int export_alloc(PxlCtx* ctx) {
  const Dev& d = ctx->d;
  const size_t nt = size_t(d.cap_tuples), nv = size_t(ctx->p.max_events) * 1024, ne = size_t(ctx->p.max_events) + 1;
  for (ExportSet& x : ctx->exp) {
    x.cap_tracks = uint32_t(nt);
    x.cap_vertices = uint32_t(nv);
    if (alloc_n(&x.index, 4 * ne) || alloc_n(&x.state, 5 * nt) || alloc_n(&x.cov, 15 * nt) || alloc_n(&x.pt, nt) ||
        alloc_n(&x.eta, nt) || alloc_n(&x.chi2, nt) || alloc_n(&x.n_hits, nt) || alloc_n(&x.vertex, nt) ||
        alloc_n(&x.tuple, nt) || alloc_n(&x.zv, nv) || alloc_n(&x.wv, nv) || alloc_n(&x.vchi2, nv) ||
        alloc_n(&x.ptv2, nv) || alloc_n(&x.ndof, nv) || alloc_n(&x.block, ne + kExpBlocks))
      return PXL_ERR_CUDA;
    for (void* q : {(void*)x.index, (void*)x.state, (void*)x.cov, (void*)x.pt, (void*)x.eta, (void*)x.chi2,
                    (void*)x.n_hits, (void*)x.vertex, (void*)x.tuple, (void*)x.zv, (void*)x.wv, (void*)x.vchi2,
                    (void*)x.ptv2, (void*)x.ndof, (void*)x.block})
      ctx->allocs.push_back(q);
    if (cudaEventCreateWithFlags(&x.ready, cudaEventDisableTiming) != cudaSuccess ||
        cudaEventCreateWithFlags(&x.copied, cudaEventDisableTiming) != cudaSuccess)
      return PXL_ERR_CUDA;
  }
  return 0;
}

int export_run(PxlCtx* ctx, const PxlExport* out, cudaStream_t s, cudaStream_t cs) {
  const Dev& d = ctx->d;
  if (!ctx->exp[0].index) {
    const int rc = export_alloc(ctx);
    if (rc) return rc;
  }
  ExportSet& x = ctx->exp[ctx->exp_next];
  ctx->exp_next ^= 1;
  const int E = ctx->last_E;
  // the set's previous copies must have left before its arrays are written again
  if (cudaStreamWaitEvent(s, ctx->last_done, 0) != cudaSuccess || cudaStreamWaitEvent(s, x.copied, 0) != cudaSuccess)
    return PXL_ERR_CUDA;
  Dev dd = d;
  dd.E = E;
  Launch L{s};
  L.pdl = E <= kPdlEvents;
  dd.pdl = L.pdl;
  const int nb = event_blocks(E, kExpBlocks, 64);
  const dim3 grid(nb, E);
  L.run(k_export_count, grid, kExpThreads, 0, dd, x);
  L.run(k_export_scan, 1, 1024, 0, dd, x, nb);
  L.run(k_export_fill, grid, kExpThreads, 0, dd, x);
  if (cudaGetLastError() != cudaSuccess || cudaEventRecord(x.ready, s) != cudaSuccess ||
      cudaStreamWaitEvent(cs, x.ready, 0) != cudaSuccess)
    return PXL_ERR_CUDA;
  if (E <= kPdlEvents && device_writable(*out, E)) {
    Launch C{cs};
    C.run(k_export_out, kExpOutBlocks, kExpThreads, 0, x, *out, E);
    return cudaGetLastError() == cudaSuccess && cudaEventRecord(x.copied, cs) == cudaSuccess ? 0 : PXL_ERR_CUDA;
  }
  const size_t mt = size_t(std::min<int64_t>(out->max_tracks, x.cap_tracks));
  const size_t mv = size_t(std::min<int64_t>(out->max_vertices, x.cap_vertices));
  auto cp = [&](void* dst, const void* src, size_t bytes) {
    return !dst || bytes == 0 || cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, cs) == cudaSuccess;
  };
  const bool ok = cp(out->index, x.index, size_t(E + 1) * 16) && cp(out->state, x.state, mt * 20) &&
                  cp(out->cov, x.cov, mt * 60) && cp(out->pt, x.pt, mt * 4) && cp(out->eta, x.eta, mt * 4) &&
                  cp(out->chi2, x.chi2, mt * 4) && cp(out->n_hits, x.n_hits, mt) && cp(out->vertex, x.vertex, mt * 2) &&
                  cp(out->tuple, x.tuple, mt * 4) && cp(out->zv, x.zv, mv * 4) && cp(out->wv, x.wv, mv * 4) &&
                  cp(out->vchi2, x.vchi2, mv * 4) && cp(out->ptv2, x.ptv2, mv * 4) && cp(out->ndof, x.ndof, mv * 4);
  if (!ok || cudaEventRecord(x.copied, cs) != cudaSuccess) return PXL_ERR_CUDA;
  return 0;
}

int64_t export_bytes(const PxlExport* out, int32_t n_events) {
  const int64_t mt = out->max_tracks, mv = out->max_vertices;
  int64_t b = out->index ? int64_t(n_events + 1) * 16 : 0;
  b += (out->state ? 20 : 0) * mt + (out->cov ? 60 : 0) * mt + (out->pt ? 4 : 0) * mt + (out->eta ? 4 : 0) * mt +
       (out->chi2 ? 4 : 0) * mt + (out->n_hits ? 1 : 0) * mt + (out->vertex ? 2 : 0) * mt + (out->tuple ? 4 : 0) * mt;
  b += ((out->zv ? 4 : 0) + (out->wv ? 4 : 0) + (out->vchi2 ? 4 : 0) + (out->ptv2 ? 4 : 0) + (out->ndof ? 4 : 0)) * mv;
  return b;
}

}  // namespace pxl

extern "C" int32_t pxl_export_async(PxlCtx* ctx, const PxlExport* out, void* stream, void* copy_stream) {
  if (!ctx || !out || out->max_tracks < 0 || out->max_vertices < 0) return PXL_ERR_ARG;
  if (ctx->last_E <= 0 || (ctx->done_mask & PXL_STAGE_VERTICES) == 0) return PXL_ERR_STATE;
  if (cudaSetDevice(ctx->p.device) != cudaSuccess) return PXL_ERR_CUDA;
  cudaStream_t s = stream ? static_cast<cudaStream_t>(stream) : ctx->stream;
  cudaStream_t cs = copy_stream ? static_cast<cudaStream_t>(copy_stream) : s;
  const int rc = pxl::export_run(ctx, out, s, cs);
  return rc ? rc : 0;
}

extern "C" int64_t pxl_export_bytes(const PxlExport* out, int32_t n_events) {
  if (!out || n_events < 0) return PXL_ERR_ARG;
  return pxl::export_bytes(out, n_events);
}
