// The plan of a segmented sort (radix_sort.cuh), built by one CTA: of a launch of its own, or of another
// kernel's launch that does not need the plan yet.
#pragma once
#include "radix_sort.cuh"
#include "scan.cuh"

namespace b200tbe {

// What build_sort_plan describes: seg_start[s] = offsets[s * stride] (clamped to n), seg_tile_base = exclusive
// prefix of the tiles per segment, then one descriptor per tile. Every thread of the CTA takes part.
__device__ __forceinline__ void plan_sort(const void* __restrict__ offsets, int offset_bytes, int num_segments,
                                          int64_t stride, int64_t n, int max_tiles, const SortPlanMem& mem,
                                          int32_t* status) {
  const int threads = static_cast<int>(blockDim.x);
  uint32_t carry = 0;
  bool ordered = true;
  auto start_of = [&](int s) -> int64_t {
    const int64_t i = static_cast<int64_t>(s) * stride;
    int64_t v = offset_bytes == 8 ? load_index<int64_t>(offsets, i) : load_index<int32_t>(offsets, i);
    if (v < 0) v = 0;
    return v > n ? n : v;
  };
  for (int base = 0; base <= num_segments; base += threads) {
    const int s = base + static_cast<int>(threadIdx.x);
    uint32_t tiles = 0;
    if (s <= num_segments) {
      const int64_t first = start_of(s);
      mem.seg_start[s] = static_cast<uint32_t>(first);
      if (s < num_segments) {
        const int64_t len = start_of(s + 1) - first;
        ordered = ordered && len >= 0;
        tiles = len > 0 ? static_cast<uint32_t>((len + kSortPlanTile - 1) / kSortPlanTile) : 0u;
      }
    }
    uint32_t total;
    const uint32_t prefix = block_exclusive_scan(tiles, &total);
    if (s <= num_segments) mem.seg_tile_base[s] = carry + prefix;
    carry += total;
  }
  // Segments that end before they begin would overlap others: no tile is in use then, so that nothing is sorted
  // and nothing done with the result. (The barrier: the segments are written.)
  if (!__syncthreads_and(ordered && carry <= static_cast<uint32_t>(max_tiles))) {
    if (threadIdx.x == 0 && status != nullptr) atomicOr(status, B200TBE_DEV_OFFSETS_NOT_MONOTONE);
    carry = 0;
  }
  if (threadIdx.x == 0) *mem.planned_tiles = *mem.total_tiles = carry;
  for (uint32_t tile = threadIdx.x; tile < carry; tile += threads) {
    // the last segment whose first tile is <= tile (empty segments share their successor's value)
    int lo = 0, hi = num_segments - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (mem.seg_tile_base[mid] <= tile) {
        lo = mid;
      } else {
        hi = mid - 1;
      }
    }
    const uint32_t first = mem.seg_tile_base[lo];
    const uint32_t begin = mem.seg_start[lo] + (tile - first) * kSortPlanTile;
    const uint32_t end = mem.seg_start[lo + 1];
    const uint32_t count = end - begin < static_cast<uint32_t>(kSortPlanTile) ? end - begin : kSortPlanTile;
    mem.tile_desc[tile] = make_uint4(begin, count, static_cast<uint32_t>(lo), first);
  }
}

}  // namespace b200tbe
