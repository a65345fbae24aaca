// Stable least-significant-digit radix sort of (key, 32-bit payload) pairs.
//
// One pass per digit of up to 10 bits, three steps per pass, none of which waits on another CTA:
//   1. per-tile digit histograms (shared-memory counters), stored digit-major: counts[d][tile];
//   2. an exclusive scan over that matrix read in storage order, which turns each entry into the
//      global position of the first key of tile `tile` with digit d;
//   3. a scatter: every warp ranks its 32 consecutive keys per round by finding the lanes with an
//      equal digit, one warp vote per digit bit (measured faster than the match instruction; keys
//      of equal digit get consecutive ranks in lane order, so the order of equal keys is kept),
//      the tile is reordered by digit in shared memory, and then written out so that keys of one
//      digit go to consecutive addresses.
// Keys and payloads are read and written exactly once per pass (plus one extra read of the keys
// for the histogram); with 25..28-bit keys that is 3 passes.
//
// Segmented form (SortPlan): the array is a sequence of independent segments (the lookups of one
// embedding table each), every tile lies inside one segment, and the digit counts are stored
// segment-major -- counts[segment][digit][tile of the segment] -- so that ONE exclusive scan over
// the whole matrix still yields global positions, while keys never leave their segment. Only the
// bits that differ inside a segment are sorted: 22 bits for tables of 4 M rows however many tables
// there are.
#include "sort_plan.cuh"

namespace b200tbe {
namespace {

constexpr int kSortThreads = 256;
constexpr int kSortWarps = kSortThreads / 32;
constexpr int kMaxRadix = 2048;        // widest digit table (segmented sort)
constexpr int kDefaultDigitBits = 10;  // widest digit of the unsegmented sort
constexpr int kFlatRadix = 1 << kDefaultDigitBits;
constexpr int kMaxDigitBits = 11;      // widest digit any pass may use

template <typename KeyT>
struct SortTile {
  static constexpr int kItems = sizeof(KeyT) == 4 ? 16 : 8;  // keys per thread
  static constexpr int kTile = kSortThreads * kItems;
};

// Where a CTA's tile lies and where its digit counts go. Flat sort: tile i is keys
// [i * kTile, ...), counts[d * num_tiles + i]. Segmented sort: read from the tile's descriptor.
struct TilePlace {
  int64_t base;
  int tile_n;
  int64_t col;     // index of digit 0's count
  int64_t stride;  // distance between consecutive digits' counts
  bool live;
  uint32_t seg_begin;            // first key of the segment
  int seg_first, seg_tiles;      // its tiles
};

// (by_tile: counts[tile][digit], for sum_counts).
template <int kTile>
__device__ __forceinline__ TilePlace place_tile(bool by_tile, int64_t n, int radix, int num_tiles, const uint4* desc,
                                                const uint32_t* seg_tile_base,
                                                const uint32_t* total_tiles) {
  TilePlace t{};
  if (desc == nullptr) {
    t.base = static_cast<int64_t>(blockIdx.x) * kTile;
    t.tile_n = n - t.base < kTile ? static_cast<int>(n - t.base) : kTile;
    t.col = blockIdx.x;
    t.stride = num_tiles;
    t.live = true;
    return t;
  }
  t.live = blockIdx.x < __ldg(total_tiles);
  if (!t.live) return t;
  const uint4 d = __ldg(desc + blockIdx.x);  // {begin, count, segment, first tile of the segment}
  t.base = d.x;
  t.tile_n = static_cast<int>(d.y);
  t.seg_first = static_cast<int>(d.w);
  t.seg_tiles = static_cast<int>(__ldg(seg_tile_base + d.z + 1) - d.w);
  t.seg_begin = d.x - (blockIdx.x - d.w) * kTile;
  t.stride = by_tile ? 1 : t.seg_tiles;
  t.col = by_tile ? static_cast<int64_t>(radix) * blockIdx.x : static_cast<int64_t>(radix) * d.w + (blockIdx.x - d.w);
  return t;
}

template <typename KeyT, bool kSum>
__global__ void __launch_bounds__(kSortThreads)
    sort_histogram_kernel(const KeyT* __restrict__ keys, int64_t n, int shift, uint32_t mask,
                          int radix, uint32_t* __restrict__ counts, int num_tiles,
                          const uint4* __restrict__ desc, const uint32_t* __restrict__ seg_tile_base,
                          const uint32_t* __restrict__ total_tiles, const SortVeto veto) {
  constexpr int kItems = SortTile<KeyT>::kItems;
  constexpr int kTile = SortTile<KeyT>::kTile;
  __shared__ uint32_t hist[kMaxRadix];
  if (sizeof(KeyT) == 4 && veto.count > 0) {   // this CTA's share of the flags (plans have 4-byte keys)
    const int64_t each = (veto.count + gridDim.x - 1) / gridDim.x;
    const int64_t last = (blockIdx.x + 1) * each < veto.count ? (blockIdx.x + 1) * each : veto.count;
    bool set = false;
    for (int64_t i = blockIdx.x * each + threadIdx.x; i < last; i += kSortThreads) set = set || __ldg(veto.flags + i) != 0;
    if (set) {
      if (veto.status != nullptr) atomicOr(veto.status, B200TBE_DEV_OFFSETS_NOT_MONOTONE);
      atomicExch(veto.total_tiles, 0u);
    }
  }
  const TilePlace tp = place_tile<kTile>(kSum, n, radix, num_tiles, desc, seg_tile_base, total_tiles);
  if (!tp.live) return;
  // all of the thread's keys are requested before the first is counted
  KeyT k[kItems];
#pragma unroll
  for (int i = 0; i < kItems; ++i) {
    const int it = i * kSortThreads + threadIdx.x;
    k[i] = it < tp.tile_n ? keys[tp.base + it] : KeyT(0);
  }
  for (int d = threadIdx.x; d < radix; d += kSortThreads) hist[d] = 0;
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kItems; ++i) {
    const int it = i * kSortThreads + threadIdx.x;
    if (it < tp.tile_n) atomicAdd(&hist[static_cast<uint32_t>(k[i] >> shift) & mask], 1u);
  }
  __syncthreads();
  for (int d = threadIdx.x; d < radix; d += kSortThreads) counts[d * tp.stride + tp.col] = hist[d];
}

// The counts of one digit in the tiles of this tile's segment, summed over the tiles before this one and over
// all of them. Where segments have few tiles this takes the place of the scan: the counts are stored tile by
// tile (a tile's digits together), a thread adds up one digit's, and two launches a pass do instead of five:
// 0.63 M pairs in 14 segments, three passes, 90 us with the gaps between launches before, 50 now.
struct DigitCounts {
  uint32_t before, all;
};
__device__ __forceinline__ DigitCounts sum_counts(const uint32_t* __restrict__ counts, const TilePlace& tp, int radix) {
  DigitCounts c{0u, 0u};
  if (static_cast<int>(threadIdx.x) >= radix) return c;
  const uint32_t* at = counts + static_cast<int64_t>(tp.seg_first) * radix + threadIdx.x;
  const int mine = static_cast<int>(blockIdx.x) - tp.seg_first;
  constexpr int kBatch = 16;
  for (int q0 = 0; q0 < tp.seg_tiles; q0 += kBatch) {
    uint32_t v[kBatch];
#pragma unroll
    for (int u = 0; u < kBatch; ++u) v[u] = q0 + u < tp.seg_tiles ? __ldg(at + (q0 + u) * radix) : 0u;
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      c.all += v[u];
      if (q0 + u < mine) c.before += v[u];
    }
  }
  return c;
}

// Shared memory of the scatter kernel: per-warp digit counters (16 bits are enough: a warp holds
// at most 32 * kItems keys, a tile at most 4096), the tile-level digit offsets, and the staging
// area in which the tile is reordered. Once the tile is staged the counters are dead and their
// space holds the per-digit distance from staging position to global position. For 4-byte keys:
// 38 KB with 256 digits, 52 KB with 1024, 72 KB with 2048 (four, four and three CTAs per SM; with 256
// digits five fit at 48 registers a thread, but the keys and ranks then spill: 3 passes over 26.7 M pairs
// 400 us, 386 with four).
template <typename KeyT, int kRadix>
struct ScatterSmem {
  union {
    uint16_t warp_hist[kSortWarps][kRadix];
    uint32_t delta[kRadix];
  };
  uint32_t digit_start[kRadix];
  KeyT keys[SortTile<KeyT>::kTile];
  uint32_t vals[SortTile<KeyT>::kTile];
};

// kRadix: capacity of the digit tables (>= radix, a multiple of kSortThreads). kBits: bits ranked (>= those
// of the pass's digit, the ones above are zero); the votes are a third of the kernel's instructions, so
// passes of 7 and 6 bits vote 7 and 6 times. kFull: the tile holds kTile keys (every tile but a segment's
// last), so no step tests a position against the tile's end. kSum: see sum_counts.
template <typename KeyT, int kRadix, int kBits, bool kFull, bool kSum>
__device__ __forceinline__ void scatter_tile(ScatterSmem<KeyT, kRadix>& sm, const TilePlace& tp,
                                             const KeyT* __restrict__ keys_in, const uint32_t* __restrict__ vals_in,
                                             KeyT* __restrict__ keys_out, uint32_t* __restrict__ vals_out,
                                             int shift, uint32_t mask, int radix,
                                             const uint32_t* __restrict__ positions) {
  constexpr int kItems = SortTile<KeyT>::kItems;
  constexpr int kTile = SortTile<KeyT>::kTile;
  constexpr int kDigitsPerThread = kRadix / kSortThreads;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  {
    uint32_t* z = reinterpret_cast<uint32_t*>(&sm.warp_hist[0][0]);
    for (int i = threadIdx.x; i < kSortWarps * kRadix / 2; i += kSortThreads) z[i] = 0;
  }

  const int64_t base = tp.base;
  const int tile_n = kFull ? kTile : tp.tile_n;
  const int warp_base = warp * (kItems * 32);
  const uint32_t lanemask_lt = (1u << lane) - 1u;

  // all of the thread's keys are requested before the first is looked at
  KeyT k[kItems];
#pragma unroll
  for (int r = 0; r < kItems; ++r) {
    const int it = warp_base + r * 32 + lane;
    k[r] = (kFull || it < tile_n) ? keys_in[base + it] : KeyT(0);
  }
  DigitCounts seg{};
  if (kSum) seg = sum_counts(positions, tp, radix);
  __syncthreads();

  // ranks inside the warp, two to a register: sixteen keys, as many payloads in flight and separate ranks spill
  uint32_t rank[kItems / 2];
#pragma unroll
  for (int r = 0; r < kItems; ++r) {
    const int it = warp_base + r * 32 + lane;
    const bool valid = kFull || it < tile_n;
    const uint32_t d = static_cast<uint32_t>(k[r] >> shift) & mask;
    // lanes holding the same digit, found one bit at a time with warp votes
    uint32_t peers = kFull ? kFullMask : __ballot_sync(kFullMask, valid);
#pragma unroll
    for (int b = 0; b < kBits; ++b) {
      const bool bit = (d >> b) & 1u;
      const uint32_t with_bit = __ballot_sync(kFullMask, bit);
      peers &= bit ? with_bit : ~with_bit;
    }
    // Every lane reads its digit's counter, then the lowest lane of each digit advances it. (Handing the
    // value from that lane to its peers with a shuffle over the peers' mask makes the warp run the
    // shuffle once per distinct digit, twenty-odd times.)
    const uint32_t before = sm.warp_hist[warp][d];
    const uint32_t my_rank = before + __popc(peers & lanemask_lt);   // < 32 * kItems
    rank[r / 2] = r & 1 ? rank[r / 2] | (my_rank << 16) : my_rank;
    __syncwarp();
    if (valid && (peers & lanemask_lt) == 0) sm.warp_hist[warp][d] = static_cast<uint16_t>(before + __popc(peers));
    __syncwarp();
  }
  __syncthreads();

  // per digit: exclusive prefix over the warps, then over the digits of the tile; thread i owns
  // the kDigitsPerThread consecutive digits starting at i * kDigitsPerThread
  uint32_t totals[kDigitsPerThread], run_total[kDigitsPerThread];
  uint32_t thread_total = 0;
#pragma unroll
  for (int j = 0; j < kDigitsPerThread; ++j) {
    const int d = threadIdx.x * kDigitsPerThread + j;
    uint32_t run = 0;
#pragma unroll
    for (int w = 0; w < kSortWarps; ++w) {
      const uint32_t c = sm.warp_hist[w][d];
      sm.warp_hist[w][d] = static_cast<uint16_t>(run);
      run += c;
    }
    run_total[j] = run;
    thread_total += run;
  }
  uint32_t unused_total;
  uint32_t start = block_exclusive_scan(thread_total, &unused_total);
  uint32_t seg_start = 0;
  if (kSum) seg_start = tp.seg_begin + block_exclusive_scan(seg.all, &unused_total);
#pragma unroll
  for (int j = 0; j < kDigitsPerThread; ++j) {
    const int d = threadIdx.x * kDigitsPerThread + j;
    sm.digit_start[d] = start;
    // global position of the tile's first key of digit d, minus its staging position
    const uint32_t at = kSum ? seg_start + seg.before : (d < radix ? positions[d * tp.stride + tp.col] : 0u);
    totals[j] = at - start;
    start += run_total[j];
  }
  __syncthreads();

#pragma unroll
  for (int r = 0; r < kItems; ++r) {
    const int it = warp_base + r * 32 + lane;
    if (kFull || it < tile_n) {
      const uint32_t d = static_cast<uint32_t>(k[r] >> shift) & mask;
      const uint32_t my_rank = r & 1 ? rank[r / 2] >> 16 : rank[r / 2] & 0xffffu;
      const uint32_t pos = sm.digit_start[d] + sm.warp_hist[warp][d] + my_rank;
      sm.keys[pos] = k[r];
      sm.vals[pos] = vals_in[base + it];
    }
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kDigitsPerThread; ++j) sm.delta[threadIdx.x * kDigitsPerThread + j] = totals[j];
  __syncthreads();

  if (kFull) {
#pragma unroll 4
    for (int i = threadIdx.x; i < kTile; i += kSortThreads) {
      const KeyT key = sm.keys[i];
      const uint32_t d = static_cast<uint32_t>(key >> shift) & mask;
      const uint32_t dst = static_cast<uint32_t>(i) + sm.delta[d];
      keys_out[dst] = key;
      vals_out[dst] = sm.vals[i];
    }
  } else {
    for (int i = threadIdx.x; i < tile_n; i += kSortThreads) {
      const KeyT key = sm.keys[i];
      const uint32_t d = static_cast<uint32_t>(key >> shift) & mask;
      const uint32_t dst = static_cast<uint32_t>(i) + sm.delta[d];
      keys_out[dst] = key;
      vals_out[dst] = sm.vals[i];
    }
  }
}

template <typename KeyT, int kRadix, int kBits, bool kSum>
__global__ void __launch_bounds__(kSortThreads, kRadix > 1024 ? 3 : 4)
    sort_scatter_kernel(const KeyT* __restrict__ keys_in, const uint32_t* __restrict__ vals_in,
                        KeyT* __restrict__ keys_out, uint32_t* __restrict__ vals_out, int64_t n,
                        int shift, uint32_t mask, int radix,
                        const uint32_t* __restrict__ positions, int num_tiles,
                        const uint4* __restrict__ desc, const uint32_t* __restrict__ seg_tile_base,
                        const uint32_t* __restrict__ total_tiles) {
  constexpr int kTile = SortTile<KeyT>::kTile;
  extern __shared__ __align__(16) unsigned char sort_smem[];
  ScatterSmem<KeyT, kRadix>& sm = *reinterpret_cast<ScatterSmem<KeyT, kRadix>*>(sort_smem);
  const TilePlace tp = place_tile<kTile>(kSum, n, radix, num_tiles, desc, seg_tile_base, total_tiles);
  if (!tp.live) return;
  if (tp.tile_n == kTile) {
    scatter_tile<KeyT, kRadix, kBits, true, kSum>(sm, tp, keys_in, vals_in, keys_out, vals_out, shift, mask, radix, positions);
  } else {
    scatter_tile<KeyT, kRadix, kBits, false, kSum>(sm, tp, keys_in, vals_in, keys_out, vals_out, shift, mask, radix, positions);
  }
}

// Up to this many segments and tiles one CTA makes the plan in one launch; beyond, it leaves the tiles to a second
// launch (4 M keys in 100 000 segments: 5.56 ms so, 5.62 in one launch; in 100 segments 400 000 keys take 66.6 us in
// one launch, 2 us more by four segments per thread).
constexpr int kOneCtaSegments = kScanThreads;
constexpr int kOneCtaTiles = 16 * kScanThreads;

template <int kItems, bool kTiles>
__global__ void __launch_bounds__(kScanThreads)
    plan_sort_kernel(const void* __restrict__ offsets, int offset_bytes, int num_segments, int64_t stride, int64_t n,
                     int max_tiles, const SortPlanMem mem, int32_t* status) {
  plan_sort<kScanThreads, kItems, kTiles>(offsets, offset_bytes, num_segments, stride, n, max_tiles, mem, status);
}

__global__ void __launch_bounds__(256) plan_tiles_kernel(int num_segments, const SortPlanMem mem) {
  const uint32_t tile = blockIdx.x * blockDim.x + threadIdx.x;
  if (tile >= *mem.total_tiles) return;
  // the last segment whose first tile is <= tile (empty segments share their successor's value)
  int lo = 0, hi = num_segments - 1;
  while (lo < hi) {
    const int mid = lo + (hi - lo + 1) / 2;
    if (__ldg(mem.seg_tile_base + mid) <= tile) {
      lo = mid;
    } else {
      hi = mid - 1;
    }
  }
  const uint32_t first = __ldg(mem.seg_tile_base + lo);
  const uint32_t begin = __ldg(mem.seg_start + lo) + (tile - first) * kSortPlanTile;
  const uint32_t left = __ldg(mem.seg_start + lo + 1) - begin;
  mem.tile_desc[tile] = make_uint4(begin, left < static_cast<uint32_t>(kSortPlanTile) ? left : kSortPlanTile,
                                   static_cast<uint32_t>(lo), first);
}

template <typename KeyT>
int64_t sort_num_tiles(int64_t n) {
  return (n + SortTile<KeyT>::kTile - 1) / SortTile<KeyT>::kTile;
}

struct PassArgs {
  int64_t n;
  int shift, bits, tiles;
  uint32_t* counts;
  const SortPlan* plan;
};

template <typename KeyT, int kRadix, int kBits, bool kSum>
int launch_scatter(const KeyT* kin, const uint32_t* vin, KeyT* kout, uint32_t* vout, const PassArgs& a,
                   cudaStream_t stream) {
  auto kernel = sort_scatter_kernel<KeyT, kRadix, kBits, kSum>;
  const size_t smem = sizeof(ScatterSmem<KeyT, kRadix>);
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           static_cast<int>(smem)) != cudaSuccess)
    return B200TBE_ERR_LAUNCH;
  const int radix = 1 << a.bits;
  kernel<<<a.tiles, kSortThreads, smem, stream>>>(
      kin, vin, kout, vout, a.n, a.shift, static_cast<uint32_t>(radix - 1), radix, a.counts,
      a.tiles, a.plan ? a.plan->tile_desc : nullptr, a.plan ? a.plan->seg_tile_base : nullptr,
      a.plan ? a.plan->total_tiles : nullptr);
  return B200TBE_OK;
}

template <typename KeyT, bool kSum>
int launch_scatter_256(const KeyT* kin, const uint32_t* vin, KeyT* kout, uint32_t* vout, const PassArgs& a,
                       cudaStream_t stream) {
  if (a.bits <= 6) return launch_scatter<KeyT, 256, 6, kSum>(kin, vin, kout, vout, a, stream);
  if (a.bits == 7) return launch_scatter<KeyT, 256, 7, kSum>(kin, vin, kout, vout, a, stream);
  return launch_scatter<KeyT, 256, 8, kSum>(kin, vin, kout, vout, a, stream);
}

// Segments whose tiles' counts are summed in the scatter kernel rather than scanned: up to this many tiles in
// all, so a segment with every key in it has no more either. There the two are even: one segment of 1 M keys
// takes three passes of 18 us scatter and nothing else, or of 12 us and three launches of 7 us; eight segments
// of 0.67 M keys took 184 us a training step scanned, 149 summed.
constexpr int64_t kSumTiles = 256;

// plan == nullptr: one flat array of n keys. Otherwise the tiles of the plan (tiles = its bound).
template <typename KeyT>
int sort_impl(KeyT* keys_a, uint32_t* vals_a, KeyT* keys_b, uint32_t* vals_b, int64_t n,
              int key_bits, int max_digit_bits, const SortPlan* plan, uint32_t* counts,
              uint32_t* tile_sums, bool* result_in_b, cudaStream_t stream) {
  const int64_t tiles64 = plan ? plan->max_tiles : sort_num_tiles<KeyT>(n);
  if (tiles64 > 0x7fffffff / (plan ? kMaxRadix : kFlatRadix)) return B200TBE_ERR_TOO_LARGE;
  const int tiles = static_cast<int>(tiles64);
  const int passes = (key_bits + max_digit_bits - 1) / max_digit_bits;
  bool in_b = false;
  int shift = 0;
  for (int pass = 0; pass < passes; ++pass) {
    // spread the bits evenly: fewer bins per pass means cheaper ranking
    const int bits = (key_bits - shift + (passes - pass) - 1) / (passes - pass);
    const int radix = 1 << bits;
    const uint32_t mask = static_cast<uint32_t>(radix - 1);
    const KeyT* kin = in_b ? keys_b : keys_a;
    const uint32_t* vin = in_b ? vals_b : vals_a;
    KeyT* kout = in_b ? keys_a : keys_b;
    uint32_t* vout = in_b ? vals_a : vals_b;
    const PassArgs a{n, shift, bits, tiles, counts, plan};
    const uint32_t* hist_tiles = plan == nullptr ? nullptr : (pass == 0 ? plan->planned_tiles : plan->total_tiles);
    const SortVeto veto = plan != nullptr && pass == 0 ? plan->veto : SortVeto{};
    const bool sum = plan != nullptr && bits <= 8 && n / kSortPlanTile <= kSumTiles;
    if constexpr (sizeof(KeyT) == 4) {   // segments have 4-byte keys
      if (sum) {
        sort_histogram_kernel<KeyT, true><<<tiles, kSortThreads, 0, stream>>>(
            kin, n, shift, mask, radix, counts, tiles, plan->tile_desc, plan->seg_tile_base, hist_tiles, veto);
        const int st = launch_scatter_256<KeyT, true>(kin, vin, kout, vout, a, stream);
        if (st != B200TBE_OK) return st;
        in_b = !in_b;
        shift += bits;
        continue;
      }
    }
    sort_histogram_kernel<KeyT, false><<<tiles, kSortThreads, 0, stream>>>(
        kin, n, shift, mask, radix, counts, tiles, plan ? plan->tile_desc : nullptr,
        plan ? plan->seg_tile_base : nullptr, hist_tiles, veto);
    // with a plan the scan starts where the first segment does, and also covers the unused tail of the matrix (tiles is an upper bound);
    // nothing reads it
    int st = exclusive_scan_u32(counts, static_cast<int64_t>(radix) * tiles, tile_sums, plan ? plan->seg_start : nullptr, stream);
    if (st != B200TBE_OK) return st;
    if (bits <= 8) {
      st = launch_scatter_256<KeyT, false>(kin, vin, kout, vout, a, stream);
    } else if (bits <= 10) {
      st = launch_scatter<KeyT, 1024, 10, false>(kin, vin, kout, vout, a, stream);
    } else {
      st = launch_scatter<KeyT, 2048, 11, false>(kin, vin, kout, vout, a, stream);
    }
    if (st != B200TBE_OK) return st;
    in_b = !in_b;
    shift += bits;
  }
  *result_in_b = in_b;
  return launch_status();
}

size_t align256(size_t x) { return (x + 255) & ~size_t{255}; }

}  // namespace

size_t radix_sort_scratch_bytes(int64_t n) {
  if (n <= 0) return 256;
  // tile count of the narrower tile (8-byte keys) bounds both key widths
  const int64_t tiles = sort_num_tiles<uint64_t>(n);
  const int64_t counts = tiles * kFlatRadix;
  return align256(static_cast<size_t>(counts) * 4) +
         align256(static_cast<size_t>(scan_num_tiles(counts)) * 4) + 256;
}

size_t radix_sort_planned_scratch_bytes(int64_t max_tiles) {
  const int64_t counts = (max_tiles > 0 ? max_tiles : 1) * kMaxRadix;
  return align256(static_cast<size_t>(counts) * 4) +
         align256(static_cast<size_t>(scan_num_tiles(counts)) * 4) + 256;
}

int64_t sort_plan_max_tiles(int64_t n, int64_t num_segments) {
  // every segment's last tile may be partial
  return n / kSortPlanTile + (num_segments > 0 ? num_segments : 0) + 1;
}

bool sort_plan_fits(int64_t max_tiles) { return max_tiles <= 0x7fffffff / kMaxRadix; }

size_t sort_plan_bytes(int64_t n, int64_t num_segments) {
  const int64_t tiles = sort_plan_max_tiles(n, num_segments);
  return 2 * align256(static_cast<size_t>(num_segments + 1) * 4) + align256(static_cast<size_t>(tiles) * sizeof(uint4)) + 256;
}

SortPlanMem sort_plan_mem(int64_t n, int64_t num_segments, void* plan_mem) {
  const int64_t tiles = sort_plan_max_tiles(n, num_segments);
  char* at = static_cast<char*>(plan_mem);
  auto take = [&](size_t bytes) {
    char* here = at;
    at += align256(bytes);
    return here;
  };
  SortPlanMem m{};
  m.seg_start = reinterpret_cast<uint32_t*>(take(static_cast<size_t>(num_segments + 1) * 4));
  m.seg_tile_base = reinterpret_cast<uint32_t*>(take(static_cast<size_t>(num_segments + 1) * 4));
  m.tile_desc = reinterpret_cast<uint4*>(take(static_cast<size_t>(tiles) * sizeof(uint4)));
  m.total_tiles = reinterpret_cast<uint32_t*>(at);
  m.planned_tiles = m.total_tiles + 1;
  return m;
}

int build_sort_plan(const void* offsets, int offset_bytes, int num_segments, int64_t stride, int64_t n,
                    void* plan_mem, int32_t* status, SortPlan* plan, cudaStream_t stream) {
  const int64_t tiles = sort_plan_max_tiles(n, num_segments);
  if (!sort_plan_fits(tiles) || num_segments < 1) return B200TBE_ERR_TOO_LARGE;
  const SortPlanMem mem = sort_plan_mem(n, num_segments, plan_mem);
  const int max_tiles = static_cast<int>(tiles);
  if (num_segments <= kOneCtaSegments && max_tiles <= kOneCtaTiles) {
    plan_sort_kernel<1, true><<<1, kScanThreads, 0, stream>>>(offsets, offset_bytes, num_segments, stride, n, max_tiles,
                                                             mem, status);
  } else {
    plan_sort_kernel<4, false><<<1, kScanThreads, 0, stream>>>(offsets, offset_bytes, num_segments, stride, n, max_tiles,
                                                              mem, status);
    plan_tiles_kernel<<<static_cast<unsigned>((tiles + 255) / 256), 256, 0, stream>>>(num_segments, mem);
  }
  *plan = sort_plan_of(mem, max_tiles);
  return launch_status();
}

int radix_sort_pairs_planned(uint32_t* keys_a, uint32_t* vals_a, uint32_t* keys_b, uint32_t* vals_b,
                             int64_t n, int key_bits, int max_digit_bits, const SortPlan& plan,
                             void* scratch, size_t scratch_bytes, bool* result_in_b,
                             cudaStream_t stream) {
  *result_in_b = false;
  if (n < 0 || key_bits < 0 || key_bits > 32 || max_digit_bits < 1 || max_digit_bits > kMaxDigitBits ||
      plan.max_tiles < 0)
    return B200TBE_ERR_BAD_ARG;
  if (n == 0 || key_bits == 0 || plan.max_tiles == 0) return B200TBE_OK;
  if (scratch == nullptr || scratch_bytes < radix_sort_planned_scratch_bytes(plan.max_tiles) ||
      !aligned_to(scratch, 256))
    return B200TBE_ERR_SCRATCH;
  uint32_t* counts = static_cast<uint32_t*>(scratch);
  uint32_t* tile_sums = reinterpret_cast<uint32_t*>(
      static_cast<char*>(scratch) + align256(static_cast<size_t>(plan.max_tiles) * kMaxRadix * 4));
  return sort_impl<uint32_t>(keys_a, vals_a, keys_b, vals_b, n, key_bits, max_digit_bits, &plan, counts,
                             tile_sums, result_in_b, stream);
}

int radix_sort_pairs(void* keys_a, uint32_t* vals_a, void* keys_b, uint32_t* vals_b, int64_t n,
                     int key_bytes, int key_bits, void* scratch, size_t scratch_bytes,
                     bool* result_in_b, cudaStream_t stream) {
  *result_in_b = false;
  if (n < 0 || key_bits < 0 || (key_bytes != 4 && key_bytes != 8) || key_bits > key_bytes * 8)
    return B200TBE_ERR_BAD_ARG;
  if (n >= (int64_t{1} << 31)) return B200TBE_ERR_TOO_LARGE;
  if (n == 0 || key_bits == 0) return B200TBE_OK;
  if (keys_a == nullptr || vals_a == nullptr || keys_b == nullptr || vals_b == nullptr)
    return B200TBE_ERR_BAD_ARG;
  if (scratch == nullptr || scratch_bytes < radix_sort_scratch_bytes(n) ||
      !aligned_to(scratch, 256))
    return B200TBE_ERR_SCRATCH;
  const int64_t tiles = sort_num_tiles<uint64_t>(n);
  uint32_t* counts = static_cast<uint32_t*>(scratch);
  uint32_t* tile_sums = reinterpret_cast<uint32_t*>(
      static_cast<char*>(scratch) + align256(static_cast<size_t>(tiles) * kFlatRadix * 4));
  if (key_bytes == 4)
    return sort_impl<uint32_t>(static_cast<uint32_t*>(keys_a), vals_a,
                               static_cast<uint32_t*>(keys_b), vals_b, n, key_bits,
                               kDefaultDigitBits, nullptr, counts, tile_sums, result_in_b, stream);
  return sort_impl<unsigned long long>(static_cast<unsigned long long*>(keys_a), vals_a,
                                       static_cast<unsigned long long*>(keys_b), vals_b, n, key_bits,
                                       kDefaultDigitBits, nullptr, counts, tile_sums, result_in_b,
                                       stream);
}

}  // namespace b200tbe

using namespace b200tbe;

extern "C" size_t b200tbe_radix_sort_scratch_bytes(int64_t n) { return radix_sort_scratch_bytes(n); }

extern "C" int b200tbe_radix_sort_pairs(void* keys_in, uint32_t* vals_in, void* keys_out,
                                        uint32_t* vals_out, int64_t n, int32_t key_bytes,
                                        int32_t key_bits, void* scratch, size_t scratch_bytes,
                                        b200tbe_stream_t stream_) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  bool in_b = false;
  const int st = radix_sort_pairs(keys_in, vals_in, keys_out, vals_out, n, key_bytes, key_bits,
                                  scratch, scratch_bytes, &in_b, stream);
  if (st != B200TBE_OK || n <= 0) return st;
  if (!in_b) {
    if (cudaMemcpyAsync(keys_out, keys_in, static_cast<size_t>(n) * key_bytes,
                        cudaMemcpyDeviceToDevice, stream) != cudaSuccess ||
        cudaMemcpyAsync(vals_out, vals_in, static_cast<size_t>(n) * 4, cudaMemcpyDeviceToDevice,
                        stream) != cudaSuccess)
      return B200TBE_ERR_LAUNCH;
  }
  return B200TBE_OK;
}

extern "C" size_t b200tbe_radix_sort_segments_scratch_bytes(int64_t n, int32_t num_segments) {
  if (n < 0 || num_segments < 0) return 0;
  return sort_plan_bytes(n, num_segments) +
         radix_sort_planned_scratch_bytes(sort_plan_max_tiles(n, num_segments));
}

extern "C" int b200tbe_radix_sort_segments(uint32_t* keys_in, uint32_t* vals_in, uint32_t* keys_out,
                                           uint32_t* vals_out, int64_t n, const void* seg_offsets,
                                           int32_t offset_bytes, int32_t num_segments, int32_t key_bits,
                                           void* scratch, size_t scratch_bytes, b200tbe_stream_t stream_) {
  if (n < 0 || num_segments < 0 || key_bits < 0 || key_bits > 32 || (offset_bytes != 4 && offset_bytes != 8))
    return B200TBE_ERR_BAD_ARG;
  if (n >= (int64_t{1} << 31)) return B200TBE_ERR_TOO_LARGE;
  if (n == 0 || num_segments == 0) return B200TBE_OK;
  if (keys_in == nullptr || vals_in == nullptr || keys_out == nullptr || vals_out == nullptr ||
      seg_offsets == nullptr)
    return B200TBE_ERR_BAD_ARG;
  if (scratch == nullptr || scratch_bytes < b200tbe_radix_sort_segments_scratch_bytes(n, num_segments) ||
      !aligned_to(scratch, 256))
    return B200TBE_ERR_SCRATCH;
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  SortPlan plan{};
  int st = build_sort_plan(seg_offsets, offset_bytes, num_segments, 1, n, scratch, nullptr, &plan, stream);
  if (st != B200TBE_OK) return st;
  char* sort_scratch = static_cast<char*>(scratch) + sort_plan_bytes(n, num_segments);
  bool in_b = false;
  st = radix_sort_pairs_planned(keys_in, vals_in, keys_out, vals_out, n, key_bits, kMaxDigitBits, plan,
                                sort_scratch, radix_sort_planned_scratch_bytes(plan.max_tiles), &in_b,
                                stream);
  if (st != B200TBE_OK) return st;
  if (!in_b) {
    if (cudaMemcpyAsync(keys_out, keys_in, static_cast<size_t>(n) * 4, cudaMemcpyDeviceToDevice, stream) !=
            cudaSuccess ||
        cudaMemcpyAsync(vals_out, vals_in, static_cast<size_t>(n) * 4, cudaMemcpyDeviceToDevice, stream) !=
            cudaSuccess)
      return B200TBE_ERR_LAUNCH;
  }
  return B200TBE_OK;
}

// ------------------------------------------------------------------------------------------------
// Sort entry point that allocates nothing.
//
// Some callers of this library cannot obtain device memory at call time: a C or C++ host that links
// libb200tbe.so directly and has no tensor allocator to borrow scratch from; a serving process that
// reserves all of HBM for embedding tables at start-up, so a later cudaMalloc may fail; and
// latency-critical loops that cannot afford the device-wide synchronisation cudaMalloc and cudaFree
// imply. For them the sort's scratch (per-tile digit counts and the scan's tile sums) lives in a
// fixed array inside the library. Every GPU that loads the library holds the array until the
// process exits, which is why the capacity is modest.
// ------------------------------------------------------------------------------------------------
namespace b200tbe {
namespace {

constexpr int64_t kStaticSortMaxPairs = int64_t{1} << 20;
// counts for the narrower (8-byte-key) tile + scan tile sums + slack, as radix_sort_scratch_bytes()
// computes for kStaticSortMaxPairs: 512 tiles x 1024 digits x 4 B = 2 MiB, plus under 4 KiB.
constexpr size_t kStaticSortScratchBytes = (size_t{512} * kFlatRadix * 4) + 4096;

static __device__ __align__(256) unsigned char g_static_sort_scratch[kStaticSortScratchBytes];

constexpr int kMaxDevices = 64;
void* g_static_sort_ptr[kMaxDevices] = {};

// The array's name is only a host-side handle; the device address has to be asked for, once per
// device, with that device current.
int static_sort_scratch(void** out) {
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return B200TBE_ERR_LAUNCH;
  void* p = __atomic_load_n(&g_static_sort_ptr[dev], __ATOMIC_ACQUIRE);
  if (p == nullptr) {
    if (cudaGetSymbolAddress(&p, g_static_sort_scratch) != cudaSuccess || p == nullptr)
      return B200TBE_ERR_LAUNCH;
    __atomic_store_n(&g_static_sort_ptr[dev], p, __ATOMIC_RELEASE);
  }
  *out = p;
  return B200TBE_OK;
}

}  // namespace
}  // namespace b200tbe

extern "C" int64_t b200tbe_radix_sort_pairs_static_max(void) { return kStaticSortMaxPairs; }

extern "C" int b200tbe_radix_sort_pairs_static(void* keys_in, uint32_t* vals_in, void* keys_out,
                                               uint32_t* vals_out, int64_t n, int32_t key_bytes,
                                               int32_t key_bits, b200tbe_stream_t stream_) {
  if (n < 0) return B200TBE_ERR_BAD_ARG;
  if (n > kStaticSortMaxPairs) return B200TBE_ERR_TOO_LARGE;
  static_assert(kStaticSortScratchBytes >= 256, "scratch too small");
  if (radix_sort_scratch_bytes(n) > kStaticSortScratchBytes) return B200TBE_ERR_TOO_LARGE;
  void* scratch = nullptr;
  const int st = static_sort_scratch(&scratch);
  if (st != B200TBE_OK) return st;
  // Nothing in the scratch has to start at zero: every pass rewrites all the counts it reads.
  return b200tbe_radix_sort_pairs(keys_in, vals_in, keys_out, vals_out, n, key_bytes, key_bits,
                                  scratch, kStaticSortScratchBytes, stream_);
}
