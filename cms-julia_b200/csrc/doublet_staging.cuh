// When the doublet count (k_doublets_count) hands a group's staged doublets to the pool.
#pragma once
#include <cstdint>

#ifndef __CUDACC__
#define __host__
#define __device__
#endif

namespace pxl {

constexpr int kGroupCells = 768;  // outer hits one 32-item group stages in shared memory

// After every step of up to 32 doublets: whether the next step might not fit any more.
__host__ __device__ constexpr bool staging_near_full(uint32_t nout) { return nout + 32 > uint32_t(kGroupCells); }

// Whether the items before `keep`, which the last staged doublet belongs to, go to the pool now; the ones before
// `done` went before. Not when one item's doublets are all there is, and not once doublets were found that the
// staging could not hold (nout counts them, the items' counts too): what is staged is then no longer the whole of
// the last item, and all items from `done` on are left to the fill pass at the group's end.
__host__ __device__ constexpr bool staging_hands_over(uint32_t nout, uint32_t keep, uint32_t done) {
  return nout <= uint32_t(kGroupCells) && keep != done;
}

}  // namespace pxl
