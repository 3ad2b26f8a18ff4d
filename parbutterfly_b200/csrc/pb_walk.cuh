// Walks over runs of slots of the ranked CSR.  Slots are 32-bit and a graph may have up to 2^32 - 2 of
// them, so a walk counts its steps (a run is shorter than 2^31) and adds them to the first slot; a
// slot is never advanced and compared with an end, which near 2^32 would wrap and not terminate.
// Plain C++ apart from the qualifier, so that it also compiles for the host.
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define PB_WALK __device__ __forceinline__
#else
#define PB_WALK inline
#endif

namespace pb {

// The steps first, first + kStride, ... of the run [beg, beg + len), four to a turn: f(slot, left) has the
// slots slot, slot + kStride, .. slot + 3 kStride, of which the r-th belongs to the run if left > r kStride.
template <int kStride, class F>
PB_WALK void walk_turns(uint32_t beg, uint32_t len, uint32_t first, F&& f) {
  uint32_t slot = beg + first;
  for (int32_t left = (int32_t)(len - first); left > 0; left -= 4 * kStride, slot += 4 * kStride) f(slot, left);
}

// Calls f(slot, valid) for the run [beg, beg + len) in groups of `group` slots, of which this is the
// one at position `at`: every caller of a group makes every call, so f may hold warp or CTA operations.
template <class F>
PB_WALK void walk_groups(uint32_t beg, uint32_t len, uint32_t group, uint32_t at, F&& f) {
  uint32_t slot = beg + at;
  for (int32_t left = (int32_t)len; left > 0; left -= (int32_t)group, slot += group) f(slot, (int32_t)at < left);
}

}  // namespace pb
