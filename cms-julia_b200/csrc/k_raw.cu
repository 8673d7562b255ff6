// FED payload walk, raw -> digi unpacking with gain calibration, and module
// starts. Restates SiPixelRawToClusterCUDA.jl:75-131 (payload walk),
// SiPixelRawToClusterGPUKernel.jl:537-658 (raw_to_digi_kernal),
// gpu_calib_pixel.jl:28-71 (calib_digis) and gpu_clustering.jl:52-74
// (count_modules) for a batch of events.
#include <cstddef>

#include "pxl_internal.cuh"

namespace pxl {

namespace {

// Single-block scan of one EvInfo count field into a base field over E events; ev[E] receives the
// batch total in both fields. With a capacity (cap >= 0), events whose region [base, base + count)
// would pass it are emptied (count = 0, buffer warning) and the batch total is capped, so that no
// later kernel indexes past the buffer.
__global__ void __launch_bounds__(1024) k_ev_scan(EvInfo* ev, int E, int count_off, int base_off, int64_t cap,
                                                  uint32_t* status) {
  pdl_sync();
  __shared__ uint32_t sh[33];
  char* base = reinterpret_cast<char*>(ev);
  uint32_t carry = 0;
  for (int b = 0; b < E; b += blockDim.x) {
    const int e = b + threadIdx.x;
    uint32_t* cnt = reinterpret_cast<uint32_t*>(base + size_t(e) * sizeof(EvInfo) + count_off);
    const uint32_t v = e < E ? *cnt : 0u;
    uint32_t tot;
    const uint32_t lo = carry + block_excl_scan(v, sh, &tot);
    if (e < E) {
      *reinterpret_cast<uint32_t*>(base + size_t(e) * sizeof(EvInfo) + base_off) = lo;
      if (cap >= 0 && int64_t(lo) + int64_t(v) > cap) {
        *cnt = 0;
        atomicOr(&ev[e].warnings, kWarnBuffer);
        atomicOr(status, kWarnBuffer);
      }
    }
    carry += tot;
  }
  if (threadIdx.x == 0) {
    *reinterpret_cast<uint32_t*>(base + size_t(E) * sizeof(EvInfo) + base_off) = carry;
    *reinterpret_cast<uint32_t*>(base + size_t(E) * sizeof(EvInfo) + count_off) =
        cap >= 0 && int64_t(carry) > cap ? uint32_t(cap) : carry;
  }
}

__device__ __forceinline__ int32_t ld_i32(const uint8_t* p) {
  // records sit on 4-byte boundaries when the blob does; read bytewise to stay safe otherwise
  uint32_t v = uint32_t(p[0]) | (uint32_t(p[1]) << 8) | (uint32_t(p[2]) << 16) | (uint32_t(p[3]) << 24);
  return int32_t(v);
}

// One block per event: FedRawDataCollection directory (bin/ReadRAW.jl:23-31), then the
// payload word counts in fedIds order (SiPixelRawToClusterCUDA.jl:75-131: skip FED 40,
// skip empty FEDs, payload = bytes [8, size-8)). The directory is a chain of records whose
// positions depend on every earlier size, so one thread follows it, a window of the event at a
// time that the whole block has just read (the chain's loads then come from L1; from L2 and with
// the slot lookup between two hops a single event's table took 44 us). The slots of the records, a
// repeated FED id's last record winning, and the FED header and trailer checks then run in parallel.
constexpr uint32_t kFedWindow = 96 * 1024;  // bytes per window
constexpr int kFedHops = 256;               // records per window

__global__ void __launch_bounds__(256) k_fed_table(Dev d, const int16_t* __restrict__ fed_slot_of) {
  pdl_sync(d);
  const int e = blockIdx.x;
  const int NF = d.n_fed_slots;
  __shared__ uint64_t s_src[kMaxFedSlots];
  __shared__ uint32_t s_nw[kMaxFedSlots];
  __shared__ int32_t s_len[kMaxFedSlots];
  __shared__ uint32_t s_last[kMaxFedSlots];  // 1 + the slot's last record so far
  __shared__ uint64_t s_pos[kFedHops];
  __shared__ int32_t s_fid[kFedHops], s_size[kFedHops];
  __shared__ uint64_t s_p;       // position of the next record
  __shared__ int32_t s_hop;      // its number
  __shared__ int s_n;            // records of the window
  __shared__ uint32_t sh[33];
  __shared__ uint32_t s_warn;
  for (int f = threadIdx.x; f < NF; f += blockDim.x) { s_nw[f] = 0; s_src[f] = 0; s_len[f] = 0; s_last[f] = 0; }
  if (threadIdx.x == 0) {
    s_warn = 0; s_p = 4; s_hop = 0;
    if (e == 0) { *d.err_count = 0; *d.status = 0; }  // of this run: set by the kernels from here on
  }
  __syncthreads();
  const uint64_t off0 = d.ev_off[e], off1 = d.ev_off[e + 1];
  const uint8_t* ev = d.raw + off0;
  const uint64_t nbytes = off1 - off0;
  const bool words = (reinterpret_cast<uintptr_t>(ev) & 3u) == 0;
  const int32_t nfeds = nbytes >= 4 ? ld_i32(ev) : 0;
  while (s_hop < nfeds) {  // the same for all threads
    const uint64_t w0 = s_p, w1 = w0 + kFedWindow < nbytes ? w0 + kFedWindow : nbytes;
    for (uint64_t q = w0 + 128u * threadIdx.x; q < w1; q += 128u * blockDim.x) {
      uint32_t v;
      asm volatile("ld.global.ca.u8 %0, [%1];" : "=r"(v) : "l"(ev + q));
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      uint64_t p = w0;
      int32_t k = s_hop;
      int n = 0;
      while (k < nfeds && n < kFedHops && (p < w1 || n == 0)) {
        if (p + 8 > nbytes) { s_warn |= kWarnBuffer; k = nfeds; break; }
        int32_t fid, size;
        if (words && (p & 3u) == 0) {
          fid = *reinterpret_cast<const int32_t*>(ev + p);
          size = *reinterpret_cast<const int32_t*>(ev + p + 4);
        } else {
          fid = ld_i32(ev + p);
          size = ld_i32(ev + p + 4);
        }
        if (size < 0 || p + 8 + uint64_t(size) > nbytes) { s_warn |= kWarnBuffer; k = nfeds; break; }
        s_pos[n] = p;
        s_fid[n] = fid;
        s_size[n] = size;
        ++n;
        ++k;
        p += 8 + uint64_t(size);
      }
      s_p = p;
      s_n = n;
      s_hop = k;
    }
    __syncthreads();
    const int r = threadIdx.x;  // kFedHops records at most, one per thread
    const int fid = r < s_n ? s_fid[r] : -1;
    const int slot = fid >= 0 && fid < 4096 ? fed_slot_of[fid] : -1;
    if (slot >= 0) atomicMax(&s_last[slot], uint32_t(r) + 1u);
    __syncthreads();
    if (slot >= 0 && s_last[slot] == uint32_t(r) + 1u) {
      const int32_t size = s_size[r];
      const uint32_t nw64 = uint32_t(size) / 8;
      s_nw[slot] = nw64 == 0 ? 0u : (size >= 16 ? uint32_t(size - 16) / 4 : 0u);
      s_src[slot] = off0 + s_pos[r] + 8 + 8;
      s_len[slot] = size;
    }
    __syncthreads();
    if (slot >= 0) s_last[slot] = 0;
    __syncthreads();
  }
  static_assert(kFedHops == 256, "one record per thread");
  // Header and trailer checks (SiPixelRawToClusterCUDA.jl:90-128, ErrorChecker.jl:82-137). The
  // reference's checker stores no error record (_includeErrors = false, ErrorChecker.jl:30-35):
  // a header failing check() ends its loop silently and a foreign source id only prints. A header
  // announcing more headers, a trailer failing check() or announcing more trailers, a
  // fragment_length other than the FED's 64-bit word count, or a size that is not a whole
  // number of 64-bit words make the reference raise; they set PXL_WARN_FED_FORMAT here and the
  // payload [8, size - 8) is unpacked as on the valid path.
  for (int f = threadIdx.x; f < NF; f += blockDim.x) {
    const int32_t len = s_len[f];
    if (len < 8) continue;  // empty FEDs are skipped (n_words == 0)
    const uint8_t* fd = d.raw + s_src[f] - 8;  // the FED's data: header, payload, trailer
    const uint32_t h0 = uint32_t(ld_i32(fd)), h1 = uint32_t(ld_i32(fd + 4));
    const uint32_t t0 = uint32_t(ld_i32(fd + len - 8)), t1 = uint32_t(ld_i32(fd + len - 4));
    bool raise = (len & 7) != 0 || len < 16;
    if ((h1 >> 28) == 0x5u && ((h0 >> 3) & 1u)) raise = true;   // more_headers (fed_header.jl:177)
    if ((t1 >> 28) != 0xAu) raise = true;                         // trailer check() (fed_trailer.jl:214)
    else if ((t1 & 0xFFFFFFu) != uint32_t(len) / 8u) raise = true;  // fragment_length (fed_trailer.jl:193)
    else if ((t0 >> 3) & 1u) raise = true;                        // more_trailers (fed_trailer.jl:201)
    if (raise) atomicOr(&s_warn, kWarnFedFormat);
  }
  uint32_t carry = 0;
  for (int b = 0; b < NF; b += blockDim.x) {
    int f = b + threadIdx.x;
    uint32_t v = f < NF ? s_nw[f] : 0u;
    uint32_t tot;
    uint32_t ex = block_excl_scan(v, sh, &tot);
    if (f < NF) {
      d.fed_src[size_t(e) * NF + f] = s_src[f];
      d.fed_nw[size_t(e) * NF + f] = v;
      d.fed_wo[size_t(e) * NF + f] = carry + ex;
    }
    carry += tot;
  }
  if (threadIdx.x == 0) {
    EvInfo& E = d.ev[e];
    E.raw_off = off0;
    E.n_words = carry;
    E.warnings = s_warn;
    E.n_errors = 0;
  }
}

// raw_to_digi_kernal + calib_digis of one FED word ww: event-local word index local, global
// digi index g, FED id fed + 1200.
__device__ __forceinline__ void unpack_word(const Dev& d, int e, uint32_t local, uint64_t g, uint8_t fed, uint32_t ww) {
  const Conditions& c = d.c;
  int16_t xx = 0, yy = 0, mid = int16_t(kInvId);
  int32_t adc = 0;
  uint32_t pdigi = 0, rawid = 0;
  d.clus[g] = int32_t(local + 1);  // count_modules: clus[i] = i
  if (ww != 0) {
    const uint32_t link = (ww >> 26) & 0x3Fu, roc = (ww >> 21) & 0x1Fu;
    const uint32_t index = uint32_t(fed) * kMaxLink * kMaxRoc + (link - 1u) * kMaxRoc + roc + 1u;  // 1-based
    // check_roc: only code 25 survives the reference's comparisons (SiPixelRawToClusterGPUKernel.jl:394-468)
    const uint8_t etype = (roc == 25u) ? 25 : 0;
    const bool skip_roc = roc < 8u ? false : (etype != 0);
    bool keep = true;
    if (d.include_errors && skip_roc) {
      uint32_t pos = atomicAdd(&d.ev[e].n_errors, 1u);
      uint32_t gp = atomicAdd(d.err_count, 1u);
      if (gp < uint32_t(d.cap_words)) {
        d.err[5 * size_t(gp) + 0] = uint32_t(e);
        d.err[5 * size_t(gp) + 1] = local;
        d.err[5 * size_t(gp) + 2] = 0xffffffffu;
        d.err[5 * size_t(gp) + 3] = ww;
        d.err[5 * size_t(gp) + 4] = 25u | (uint32_t(fed) << 8);
      }
      (void)pos;
      keep = false;
    }
    uint64_t cab = 0;
    if (keep) {
      if (index < 1u || index > kCablingSize) { atomic_or_warn(&d.ev[e], kWarnModules); keep = false; }
      else cab = c.cab[index - 1];
    }
    if (keep && d.use_quality && ((cab >> 56) & 1u)) keep = false;
    if (keep) {
      const uint32_t raw_id = uint32_t(cab);
      const bool barrel = ((raw_id >> 25) & 0x7u) == 1u;
      const uint32_t layer = barrel ? ((raw_id >> 20) & 0xFu) : 0u;
      const uint32_t the_module = barrel ? ((raw_id >> 2) & 0x3FFu) : 0u;
      const uint32_t panel = barrel ? 0u : ((raw_id >> 10) & 0x3u);
      const int side = barrel ? ((the_module < 5u) ? -1 : 1) : ((panel == 1u) ? -1 : 1);
      const uint32_t roc_in_det = uint32_t((cab >> 48) & 0xFFu);
      int32_t row, col;
      bool conv_err = false;
      if (layer == 1u) {
        col = int32_t((ww >> 15) & 0x3Fu);
        row = int32_t((ww >> 8) & 0x7Fu);
        if (d.include_errors && !(row < 80 && col < 52)) conv_err = true;
      } else {
        const int32_t dcol = int32_t((ww >> 16) & 0x1Fu), pxid = int32_t((ww >> 8) & 0xFFu);
        row = 80 - pxid / 2;
        col = dcol * 2 + pxid % 2;
        if (row < 0) { atomic_or_warn(&d.ev[e], kWarnModules); keep = false; }
        else if (d.include_errors && !((dcol < 26) & (2 <= pxid) & (pxid < 162))) conv_err = true;
      }
      if (keep && conv_err) {
        atomicAdd(&d.ev[e].n_errors, 1u);
        uint32_t gp = atomicAdd(d.err_count, 1u);
        if (gp < uint32_t(d.cap_words)) {
          d.err[5 * size_t(gp) + 0] = uint32_t(e);
          d.err[5 * size_t(gp) + 1] = local;
          d.err[5 * size_t(gp) + 2] = raw_id;
          d.err[5 * size_t(gp) + 3] = ww;
          d.err[5 * size_t(gp) + 4] = 37u | (uint32_t(fed) << 8);
        }
        keep = false;
      }
      if (keep) {
        // frame_conversion, SiPixelRawToClusterGPUKernel.jl:271-350
        int32_t sr, sc, ro, co;
        const bool flip = barrel ? (side == -1 && layer != 1u) : true;
        if (flip) {
          if (roc_in_det < 8u) { sr = 1; sc = -1; ro = 0; co = (8 - int32_t(roc_in_det)) * 52 - 1; }
          else { sr = -1; sc = 1; ro = 159; co = (int32_t(roc_in_det) - 8) * 52; }
        } else {
          if (roc_in_det < 8u) { sr = -1; sc = 1; ro = 159; co = int32_t(roc_in_det) * 52; }
          else { sr = 1; sc = -1; ro = 0; co = (16 - int32_t(roc_in_det)) * 52 - 1; }
        }
        const int32_t grow = sr * row + ro, gcol = sc * col + co;
        if (grow < 0 || gcol < 0) {
          atomic_or_warn(&d.ev[e], kWarnModules);
        } else {
          xx = int16_t(grow);
          yy = int16_t(gcol);
          adc = int32_t(ww & 0xFFu);
          const uint32_t a = uint32_t(adc) < 1023u ? uint32_t(adc) : 1023u;
          pdigi = uint32_t(grow) | (uint32_t(gcol) << 11) | (a << 22);
          mid = int16_t(uint32_t(cab >> 32) & 0xFFFFu);
          rawid = raw_id;
          // calib_digis, gpu_calib_pixel.jl:41-70, with get_ped_and_gain
          if (mid != int16_t(kInvId) && (mid < 0 || mid >= kMaxNumModules)) {
            atomic_or_warn(&d.ev[e], kWarnModules);  // the reference indexes its 2000-entry gain table out of range
            mid = int16_t(kInvId);
          }
          if (mid != int16_t(kInvId)) {
            const float cf = mid < 96 ? 50.f : 47.f;
            const float off = mid < 96 ? -670.f : -60.f;
            const int m = mid;
            const uint32_t offset = c.gain_first[m] + uint32_t(int32_t(yy)) * c.gain_lcd[m] +
                                    2u * (uint32_t(int32_t(xx)) / c.rows_avg);
            const uint32_t kk = offset / 2;
            if (kk >= c.n_gain_pairs) {
              atomic_or_warn(&d.ev[e], kWarnModules);
            } else {
              const uint16_t pr = c.gain_pairs[kk];
              const uint32_t sg = pr & 0xFFu, sp = pr >> 8;
              const bool bad = sp == c.dead_flag || sp == c.noisy_flag;
              const float ped = __fadd_rn(__fmul_rn(float(sp), c.ped_prec), c.min_ped);
              const float gain = __fadd_rn(__fmul_rn(float(sg), c.gain_prec), c.min_gain);
              if (bad) {
                mid = int16_t(kInvId);
                adc = 0;
              } else {
                const float vcal = __fsub_rn(__fmul_rn(float(adc), gain), __fmul_rn(ped, gain));
                const float v = __fadd_rn(__fmul_rn(vcal, cf), off);
                const int32_t t = int32_t(truncf(v));
                adc = t > 100 ? t : 100;
              }
            }
          }
        }
      }
    }
  }
  d.xx[g] = xx; d.yy[g] = yy; d.adc[g] = adc; d.mid[g] = mid; d.pdigi[g] = pdigi; d.rawid[g] = rawid;
}

// raw_to_digi_kernal + calib_digis for the words of one FED slot per `parts` warps (a FED holds a
// few hundred words, which one warp decodes in a few steps; in a small batch, where the slots do not
// fill the GPU, its steps go to several warps: 78 us for one event of pileup 50 with one). The payload
// is read with 128-bit loads where it sits on 4-byte boundaries (always, for FED sizes in whole
// 64-bit words): the words before the first 16-byte boundary and after the last one are read
// singly, the rest as 16-byte vectors.
constexpr int kUnpackWarps = 8;

__global__ void __launch_bounds__(32 * kUnpackWarps) k_unpack(Dev d, uint32_t parts) {
  pdl_sync(d);
  __shared__ __align__(16) uint32_t s_words[kUnpackWarps][128];
  const unsigned lane = threadIdx.x & 31u, wq = threadIdx.x >> 5;
  const uint32_t wid = blockIdx.x * kUnpackWarps + wq, part = wid % parts;
  const int f = int(wid / parts), e = blockIdx.y;
  const int NF = d.n_fed_slots;
  if (f >= NF) return;
  const size_t fs = size_t(e) * NF + f;
  const uint32_t nw = d.fed_nw[fs];
  if (nw == 0) return;
  const EvInfo& E = d.ev[e];
  const uint32_t wo = d.fed_wo[fs];
  const uint64_t gbase = uint64_t(E.word_base) + wo;
  if (gbase + nw > uint64_t(d.cap_words)) {
    if (lane == 0) { atomic_or_warn(&d.ev[e], kWarnBuffer); atomicOr(d.status, kWarnBuffer); }
    return;
  }
  const uint8_t* src = d.raw + d.fed_src[fs];
  const uint8_t fed = uint8_t(d.c.fed_ids[f] - 1200u);
  // The reference stores one FED id per word pair (initialize_word_fed,
  // SiPixelRawToClusterGPUKernel.jl:217-226): a FED ending on an odd word leaves its last word in
  // a pair that the next non-empty FED writes (or none: id 0). Only FED sizes that are not whole
  // 64-bit words, on which the reference raises, give odd word counts.
  uint8_t fed_last = fed;
  if ((wo + nw) & 1u) {
    fed_last = 0;
    for (int f2 = f + 1; f2 < NF; ++f2)
      if (d.fed_nw[size_t(e) * NF + f2] > 0) { fed_last = uint8_t(d.c.fed_ids[f2] - 1200u); break; }
  }
  auto word = [&](uint32_t k, uint32_t ww) {
    unpack_word(d, e, wo + k, gbase + k, k + 1 == nw ? fed_last : fed, ww);
  };
  if ((reinterpret_cast<uintptr_t>(src) & 3u) == 0) {
    const uint32_t* src32 = reinterpret_cast<const uint32_t*>(src);
    uint32_t head = uint32_t((16u - (reinterpret_cast<uintptr_t>(src) & 15u)) & 15u) >> 2;
    head = head < nw ? head : nw;
    if (part == 0 && lane < head) word(lane, __ldg(src32 + lane));
    const uint32_t nvec = (nw - head) >> 2;
    const uint4* v = reinterpret_cast<const uint4*>(src32 + head);
    // the warp loads 32 aligned 16-byte vectors (128 words) and decodes them word by word through
    // shared memory, lane l taking words l, l + 32, l + 64, l + 96, so that the per-digi stores
    // of consecutive lanes stay consecutive
    uint32_t* sw = s_words[wq];
    for (uint32_t j0 = 32 * part; j0 < nvec; j0 += 32 * parts) {
      if (j0 + lane < nvec) reinterpret_cast<uint4*>(sw)[lane] = __ldg(v + j0 + lane);
      __syncwarp();
      const uint32_t nwords = 4u * min(32u, nvec - j0);
#pragma unroll
      for (uint32_t i = 0; i < 4; ++i) {
        const uint32_t wi = 32u * i + lane;
        if (wi < nwords) word(head + 4u * j0 + wi, sw[wi]);
      }
      __syncwarp();
    }
    if (part == 0)
      for (uint32_t k = head + 4 * nvec + lane; k < nw; k += 32) word(k, __ldg(src32 + k));
  } else {
    for (uint32_t k = 32 * part + lane; k < nw; k += 32 * parts) {
      uint32_t ww;
      memcpy(&ww, src + 4ull * k, 4);
      word(k, ww);
    }
  }
}

// count_modules flag: a valid digi whose previous valid digi (in the event) has another id.
__device__ __forceinline__ bool module_start_flag(const Dev& d, uint64_t ebase, uint32_t i) {
  const int16_t id = d.mid[ebase + i];
  if (id == int16_t(kInvId)) return false;
  int64_t j = int64_t(i) - 1;
  while (j >= 0 && d.mid[ebase + j] == int16_t(kInvId)) --j;
  return j < 0 || d.mid[ebase + j] != id;
}

// Module starts per FED slot, `parts` warps per slot, each a range of its words (one warp where
// the batch's slots fill the GPU): the flags of 32 words per step, counted with a ballot.
constexpr int kModWarps = 8;

__device__ __forceinline__ uint2 part_words(uint32_t nw, uint32_t part, uint32_t parts) {
  const uint32_t len = ((nw + parts - 1) / parts + 31u) & ~31u;
  return make_uint2(min(nw, part * len), min(nw, (part + 1) * len));
}

__global__ void __launch_bounds__(32 * kModWarps) k_modstart_count(Dev d, uint32_t parts) {
  pdl_sync(d);
  const uint32_t wid = blockIdx.x * kModWarps + (threadIdx.x >> 5);
  const int f = int(wid / parts), e = blockIdx.y;
  const int NF = d.n_fed_slots;
  if (f >= NF) return;
  const unsigned lane = threadIdx.x & 31u;
  const size_t fs = size_t(e) * NF + f;
  const uint32_t nw = d.fed_nw[fs], wo = d.fed_wo[fs];
  const uint2 r = part_words(nw, wid % parts, parts);
  uint32_t cnt = 0;
  const uint64_t ebase = d.ev[e].word_base;
  if (ebase + wo + nw <= uint64_t(d.cap_words))
    for (uint32_t k0 = r.x; k0 < r.y; k0 += 32) {
      const uint32_t k = k0 + lane;
      cnt += __popc(__ballot_sync(0xffffffffu, k < r.y && module_start_flag(d, ebase, wo + k)));
    }
  if (lane == 0) d.fed_nmod[fs * parts + wid % parts] = cnt;
}

// per event: module-start offsets per part of a FED slot, n_modules; zero the cluster counters
__global__ void k_modstart_scan(Dev d, uint32_t parts) {
  pdl_sync(d);
  const int e = blockIdx.x;
  const int NF = d.n_fed_slots * int(parts);
  __shared__ uint32_t sh[33];
  uint32_t carry = 0;
  for (int b = 0; b < NF; b += blockDim.x) {
    int f = b + threadIdx.x;
    uint32_t v = f < NF ? d.fed_nmod[size_t(e) * NF + f] : 0u;
    uint32_t tot;
    uint32_t ex = block_excl_scan(v, sh, &tot);
    if (f < NF) d.fed_nmod[size_t(e) * NF + f] = carry + ex;
    carry += tot;
  }
  uint32_t* cim = d.clus_in_module + size_t(e) * kMaxNumModules;
  for (int i = threadIdx.x; i < kMaxNumModules; i += blockDim.x) cim[i] = 0;
  for (int i = threadIdx.x; i < 64; i += blockDim.x) d.id_seen[size_t(e) * 64 + i] = 0;
  if (e == 0 && threadIdx.x < kListHeader) d.big_list[threadIdx.x] = 0;  // the clustering's work lists
  if (threadIdx.x == 0) {
    d.ev[e].repeated_ids = 0;
    uint32_t nm = carry < uint32_t(kMaxNumModules) ? carry : uint32_t(kMaxNumModules);
    d.ev[e].n_modules = nm;
    d.module_start[size_t(e) * (kMaxNumModules + 1)] = nm;
    d.module_start[size_t(e) * (kMaxNumModules + 1) + kMaxNumModules] = 0;
    d.clus_module_start[size_t(e) * (kMaxNumModules + 1)] = 0;
    if (carry > uint32_t(kMaxNumModules)) atomic_or_warn(&d.ev[e], kWarnModules);
  }
}

// The module starts of each part of a FED slot at the part's offset, one warp per part, in word
// order (rank of a flag = flags of the earlier lanes plus those of the earlier steps).
__global__ void __launch_bounds__(32 * kModWarps) k_modstart_fill(Dev d, uint32_t parts) {
  pdl_sync(d);
  const uint32_t wid = blockIdx.x * kModWarps + (threadIdx.x >> 5);
  const int f = int(wid / parts), e = blockIdx.y;
  const int NF = d.n_fed_slots;
  if (f >= NF) return;
  const unsigned lane = threadIdx.x & 31u;
  const unsigned lt = (1u << lane) - 1u;
  const size_t fs = size_t(e) * NF + f;
  const uint32_t nw = d.fed_nw[fs], wo = d.fed_wo[fs];
  const uint64_t ebase = d.ev[e].word_base;
  if (ebase + wo + nw > uint64_t(d.cap_words)) return;
  const uint2 range = part_words(nw, wid % parts, parts);
  uint32_t carry = d.fed_nmod[fs * parts + wid % parts];
  uint32_t* ms = d.module_start + size_t(e) * (kMaxNumModules + 1);
  for (uint32_t k0 = range.x; k0 < range.y; k0 += 32) {
    const uint32_t k = k0 + lane;
    const bool fl = k < range.y && module_start_flag(d, ebase, wo + k);
    const uint32_t bal = __ballot_sync(0xffffffffu, fl);
    if (fl) {
      const uint32_t r = carry + __popc(bal & lt);
      const uint32_t i1 = wo + k + 1;  // 1-based digi index
      // a module id starting a second run: the event's charge cut runs in serial order
      const uint16_t id = uint16_t(d.mid[ebase + wo + k]);
      if (id < 2048u) {
        const uint32_t bit = 1u << (id & 31u);
        if (atomicOr(&d.id_seen[size_t(e) * 64 + (id >> 5)], bit) & bit) d.ev[e].repeated_ids = 1;
      }
      if (r < uint32_t(kMaxNumModules - 1)) ms[r + 1] = i1;
      else atomicMax(&ms[kMaxNumModules], i1);
    }
    carry += __popc(bal);
  }
}

}  // namespace

void launch_raw(const Dev& d, const Launch& L, const int16_t* fed_slot_of) {
  const int NF = d.n_fed_slots;
  L.mark("start");
  L.run(k_fed_table, d.E, 256, 0, d, fed_slot_of);
  launch_ev_scan(d, L, int(offsetof(EvInfo, n_words)), int(offsetof(EvInfo, word_base)), d.cap_words);
  L.mark("fed_table");
  // warps per FED slot: one, more in a batch whose slots give an SM less than a wave of warps
  const int parts = event_blocks(d.E * NF, kFedParts, 16);
  L.run(k_unpack, dim3(div_up(int64_t(NF) * parts, kUnpackWarps), d.E), 32 * kUnpackWarps, 0, d, uint32_t(parts));
  L.mark("unpack_calib");
  launch_modstart(d, L, parts);
  L.mark("module_starts");
}

void launch_modstart(const Dev& d, const Launch& L, int parts) {
  const dim3 gm(div_up(int64_t(d.n_fed_slots) * parts, kModWarps), d.E);
  L.run(k_modstart_count, gm, 32 * kModWarps, 0, d, uint32_t(parts));
  L.run(k_modstart_scan, d.E, 256, 0, d, uint32_t(parts));
  L.run(k_modstart_fill, gm, 32 * kModWarps, 0, d, uint32_t(parts));
}

void launch_ev_scan(const Dev& d, const Launch& L, int count_off, int base_off, int64_t cap) {
  L.run(k_ev_scan, 1, 1024, 0, d.ev, d.E, count_off, base_off, cap, d.status);
}

}  // namespace pxl
