// The plan of a segmented sort (radix_sort.cuh), built by one CTA: of a launch of its own, or of another
// kernel's launch that does not need the plan yet.
#pragma once
#include "radix_sort.cuh"
#include "scan.cuh"

namespace b200tbe {

// What build_sort_plan describes: seg_start[s] = offsets[s * stride] (clamped to [0, n]), seg_tile_base =
// exclusive prefix of the tiles per segment, then (kTiles) one descriptor per tile. Every thread of the CTA takes
// part, kThreads of them. Segments go by batches of kItems per thread: a batch's offsets are one memory round
// trip, and a tile finds its segment by a search of the batch in shared memory. In the linearise launch four per
// thread: a training step over 8000 tables of 16 bags 639 us with one segment per thread and a search in global
// memory, 600 so; over 2000 of 64, 333 and 326.
template <int kThreads, int kItems, bool kTiles>
__device__ __forceinline__ void plan_sort(const void* __restrict__ offsets, int offset_bytes, int num_segments,
                                          int64_t stride, int64_t n, int max_tiles, const SortPlanMem& mem,
                                          int32_t* status) {
  constexpr int kBatch = kThreads * kItems;
  __shared__ uint32_t first_tile[kTiles ? kBatch : 1];      // of the batch's segments
  __shared__ uint32_t begin_of[kTiles ? kBatch + 1 : 1];
  auto start_of = [&](int64_t s) -> uint32_t {
    const int64_t i = s * stride;
    int64_t v = offset_bytes == 8 ? load_index<int64_t>(offsets, i) : load_index<int32_t>(offsets, i);
    if (v < 0) v = 0;
    return static_cast<uint32_t>(v > n ? n : v);
  };
  uint32_t carry = 0;
  bool ordered = true;
  for (int64_t base = 0; base < num_segments; base += kBatch) {
    const int place = static_cast<int>(threadIdx.x) * kItems;
    const int64_t s0 = base + place;
    uint32_t start[kItems + 1], tiles[kItems], mine = 0;
#pragma unroll
    for (int k = 0; k <= kItems; ++k) start[k] = start_of(s0 + k < num_segments ? s0 + k : num_segments);
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
      ordered = ordered && start[k] <= start[k + 1];
      const uint32_t len = start[k] < start[k + 1] ? start[k + 1] - start[k] : 0u;
      tiles[k] = (len + kSortPlanTile - 1) / kSortPlanTile;
      mine += tiles[k];
    }
    uint32_t total;
    uint32_t at = carry + block_exclusive_scan(mine, &total);
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
      if (kTiles) {
        first_tile[place + k] = at;
        begin_of[place + k] = start[k];
      }
      if (s0 + k < num_segments) {
        mem.seg_start[s0 + k] = start[k];
        mem.seg_tile_base[s0 + k] = at;
      }
      at += tiles[k];
    }
    carry += total;
    if (!kTiles) continue;
    if (threadIdx.x == kThreads - 1) begin_of[kBatch] = start[kItems];
    __syncthreads();
    const int segments = num_segments - base < kBatch ? static_cast<int>(num_segments - base) : kBatch;
    const uint32_t limit = carry < static_cast<uint32_t>(max_tiles) ? carry : static_cast<uint32_t>(max_tiles);
    for (uint32_t tile = carry - total + threadIdx.x; tile < limit; tile += kThreads) {
      // the last segment whose first tile is <= tile (empty segments share their successor's value)
      int lo = 0, hi = segments - 1;
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (first_tile[mid] <= tile) {
          lo = mid;
        } else {
          hi = mid - 1;
        }
      }
      const uint32_t first = first_tile[lo];
      const uint32_t begin = begin_of[lo] + (tile - first) * kSortPlanTile;
      const uint32_t left = begin_of[lo + 1] - begin;
      const uint32_t count = left < static_cast<uint32_t>(kSortPlanTile) ? left : kSortPlanTile;
      mem.tile_desc[tile] = make_uint4(begin, count, static_cast<uint32_t>(base + lo), first);
    }
    __syncthreads();   // the batch's arrays may be written again
  }
  // Segments that end before they start would overlap others: no tile is in use then, so that nothing is sorted
  // and nothing done with the result.
  const bool good = __syncthreads_and(ordered && carry <= static_cast<uint32_t>(max_tiles));
  if (threadIdx.x == 0) {
    mem.seg_start[num_segments] = start_of(num_segments);
    mem.seg_tile_base[num_segments] = carry;
    *mem.planned_tiles = *mem.total_tiles = good ? carry : 0u;
    if (!good && status != nullptr) atomicOr(status, B200TBE_DEV_OFFSETS_NOT_MONOTONE);
  }
}

}  // namespace b200tbe
