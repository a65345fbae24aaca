// Segment permutation of jagged data: output segment j is input segment perm[j], copied whole.
// This is the data movement of the input distribution of a table-wise sharded lookup (ids arrive
// grouped by source rank and have to be regrouped by table) and of FBGEMM's permute_2D_sparse_data.
//
// Segments range from empty bags to whole tables, so the work is split by output ELEMENT, not by
// segment: a CTA owns a tile of consecutive output elements, finds the segment of its first element
// by a CTA-wide 256-ary search over the output offsets (256 segments or fewer: none needed), lists the
// segments of the tile in shared memory once, each as the distance from its output to its input position,
// and marks which of them holds each element of the tile (first elements marked, a running maximum spreads
// the marks). Then every thread copies elements, eight loads in flight. A tile inside one segment -- most
// tiles, where whole tables move -- needs no map at all. Ids and their per-sample weights go through one
// launch: the second array costs its bytes only, not another search and map.
//
// Bound by memory: 26.7 M ids of 8 bytes and as many 4-byte weights in 128 segments take
// 108 us (5.9 TB/s); in two launches that built a map for every tile it was 92 + 69 us.
#include <assert.h>

#include <type_traits>

#include "common.cuh"

namespace b200tbe {
namespace {

constexpr int kPermThreads = 256;
constexpr int kPermItems = 16;                       // elements per thread
constexpr int kPermTile = kPermThreads * kPermItems;
constexpr int kPermMaxSegs = 2048;                  // segment boundaries a tile keeps in shared memory

template <typename OffT>
__device__ __forceinline__ int64_t load_off(const void* p, int64_t i) {
  return static_cast<int64_t>(reinterpret_cast<const OffT*>(p)[i]);
}

// Largest s in [0, n) with off[s] <= x (off is non-decreasing, off[0] <= x).
template <typename OffT>
__device__ __forceinline__ int64_t segment_of(const void* off, int64_t n, int64_t x) {
  int64_t lo = 0, hi = n - 1;
  while (lo < hi) {
    const int64_t mid = (lo + hi + 1) >> 1;
    if (load_off<OffT>(off, mid) <= x) {
      lo = mid;
    } else {
      hi = mid - 1;
    }
  }
  return lo;
}

struct NoElem {};   // no second array

// Output segment j is input segment perm[j], which starts at in_offsets[perm[j]] (kStarts: in_offsets[j] is
// already the start of segment j's source, and perm is not read).
template <typename ElemT, typename Elem2T, typename OffT, typename PermT, bool kStarts>
__global__ void __launch_bounds__(kPermThreads)
    permute_segments_kernel(const ElemT* __restrict__ in, ElemT* __restrict__ out, const Elem2T* __restrict__ in2,
                            Elem2T* __restrict__ out2, const void* __restrict__ in_offsets,
                            const void* __restrict__ out_offsets, const PermT* __restrict__ perm,
                            int64_t num_segments, int64_t total) {
  constexpr bool kTwo = !std::is_same<Elem2T, NoElem>::value;
  // the tile's k-th segment: input position minus output position of its elements
  __shared__ int64_t seg_delta[kPermMaxSegs];
  __shared__ __align__(16) uint16_t slot_of[kPermTile];   // listed segment of each element
  __shared__ int warp_live[kPermThreads / 32];
  __shared__ int warp_carry[kPermThreads / 32];
  __shared__ int64_t first_seg;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t tile0 = static_cast<int64_t>(blockIdx.x) * kPermTile;
  const int64_t tile1 = tile0 + kPermTile < total ? tile0 + kPermTile : total;
  auto source_of = [&](int64_t seg) {
    return load_off<OffT>(in_offsets, kStarts ? seg : static_cast<int64_t>(perm[seg]));
  };
  int64_t s = 0;
  if (num_segments > kPermThreads) {
    // the segment of the tile's first element, searched by the whole CTA: 256 probes per round
    // narrow the range 256-fold, so 22 bits of segments take 3 dependent loads instead of 22
    int64_t lo = 0, n = num_segments;
    while (n > 1) {
      const int64_t step = (n + kPermThreads - 1) / kPermThreads;
      const int64_t probe = (static_cast<int64_t>(threadIdx.x) + 1) * step;
      const bool le = probe < n && load_off<OffT>(out_offsets, lo + probe) <= tile0;
      const int64_t c = __syncthreads_count(le);   // the offsets are sorted: the true probes are the first c
      lo += c * step;
      n = n - c * step < step ? n - c * step : step;
    }
    if (threadIdx.x == 0) first_seg = lo;
    __syncthreads();
    s = first_seg;
  }
  {
    uint4* z = reinterpret_cast<uint4*>(slot_of);
    for (int q = threadIdx.x; q < kPermTile / 8; q += kPermThreads) z[q] = make_uint4(0u, 0u, 0u, 0u);
  }
  // the non-empty segments that intersect the tile, in order; threads take candidates round-robin
  // and a segment's slot is its rank among the non-empty ones, found with a block-wide count. Every
  // segment marks its first element with its slot (slots grow with the position).
  int filled = 0;
  bool overflow = false;
  while (true) {
    const int64_t cand = s + threadIdx.x;
    bool live = false, past = true;
    int64_t o0 = 0;
    if (cand < num_segments) {
      o0 = load_off<OffT>(out_offsets, cand);
      const int64_t o1 = load_off<OffT>(out_offsets, cand + 1);
      live = o0 < tile1 && o1 > o0 && o1 > tile0;
      past = o1 >= tile1;
    }
    const unsigned ballot = __ballot_sync(kFullMask, live);
    if (lane == 0) warp_live[warp] = __popc(ballot);
    // done when the round reached the end of the segments or the tile (also: slot_of is clear)
    const bool last_round = __syncthreads_or(threadIdx.x == kPermThreads - 1 && past);
    int before = 0, round_total = 0;
    for (int w = 0; w < kPermThreads / 32; ++w) {
      if (w < warp) before += warp_live[w];
      round_total += warp_live[w];
    }
    const int slot = filled + before + __popc(ballot & ((1u << lane) - 1u));
    if (live && slot < kPermMaxSegs) {
      seg_delta[slot] = source_of(cand) - o0;
      const int64_t at = o0 - tile0;
      slot_of[at > 0 ? at : 0] = static_cast<uint16_t>(slot);
    }
    filled += round_total;
    overflow = filled > kPermMaxSegs;
    __syncthreads();
    if (last_round || overflow) break;
    s += kPermThreads;
  }
  // offsets that end before `total` leave the rest of the output as it is
  const int64_t end = load_off<OffT>(out_offsets, num_segments);
  const int64_t live1 = tile1 < end ? tile1 : end;
  if (filled > 1 && !overflow) {
    // a running maximum over the tile spreads the marks: thread t scans elements [16 t, 16 t + 16); the
    // carry across threads is a warp / CTA max-scan
    uint4* mine = reinterpret_cast<uint4*>(slot_of + threadIdx.x * kPermItems);
    static_assert(kPermItems == 16, "two 16-byte words of marks per thread");
    uint4 m[2] = {mine[0], mine[1]};
    uint16_t* e = reinterpret_cast<uint16_t*>(m);
    int run = 0;
#pragma unroll
    for (int j = 0; j < kPermItems; ++j) run = max(run, static_cast<int>(e[j]));
    int incl = run;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int up = __shfl_up_sync(kFullMask, incl, o);
      if (lane >= o) incl = max(incl, up);
    }
    if (lane == 31) warp_carry[warp] = incl;
    __syncthreads();
    int carry = __shfl_up_sync(kFullMask, incl, 1);
    if (lane == 0) carry = 0;
    for (int w = 0; w < warp; ++w) carry = max(carry, warp_carry[w]);
#pragma unroll
    for (int j = 0; j < kPermItems; ++j) {
      carry = max(carry, static_cast<int>(e[j]));
      e[j] = static_cast<uint16_t>(carry);
    }
    mine[0] = m[0];
    mine[1] = m[1];
    __syncthreads();
  }
  const bool one = filled == 1;
  const int64_t one_delta = seg_delta[0];
  // eight elements at a time: their source positions first, then all loads, then the stores
  constexpr int kBatch = 8;
#pragma unroll
  for (int k0 = 0; k0 < kPermItems; k0 += kBatch) {
    int64_t src[kBatch];
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      const int e = (k0 + u) * kPermThreads + threadIdx.x;
      const int64_t i = tile0 + e;
      src[u] = -1;
      if (i >= live1) continue;
      if (one) {
        src[u] = i + one_delta;
      } else if (!overflow) {
        src[u] = i + seg_delta[slot_of[e]];
      } else {
        // more segment boundaries in one tile than the table holds (thousands of one-element
        // segments): every element searches the global offsets itself
        // (the last segment that starts at or before i is the non-empty one that holds it)
        const int64_t seg = segment_of<OffT>(out_offsets, num_segments, i);
        src[u] = source_of(seg) + (i - load_off<OffT>(out_offsets, seg));
      }
    }
    ElemT v[kBatch];
    Elem2T v2[kTwo ? kBatch : 1];
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      if (src[u] < 0) continue;
      v[u] = in[src[u]];
      if constexpr (kTwo) v2[u] = in2[src[u]];
    }
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      if (src[u] < 0) continue;
      const int64_t i = tile0 + static_cast<int64_t>(k0 + u) * kPermThreads + threadIdx.x;
      out[i] = v[u];
      if constexpr (kTwo) out2[i] = v2[u];
    }
  }
}

template <typename ElemT, typename Elem2T, typename OffT, typename PermT, bool kStarts>
int launch_perm(const void* in, void* out, const void* in2, void* out2, const void* in_offsets,
                const void* out_offsets, const void* perm, int64_t num_segments, int64_t total,
                cudaStream_t stream) {
  const int64_t ctas = (total + kPermTile - 1) / kPermTile;
  if (ctas > 0x7fffffff) return B200TBE_ERR_TOO_LARGE;
  permute_segments_kernel<ElemT, Elem2T, OffT, PermT, kStarts><<<static_cast<unsigned>(ctas), kPermThreads, 0, stream>>>(
      static_cast<const ElemT*>(in), static_cast<ElemT*>(out), static_cast<const Elem2T*>(in2),
      static_cast<Elem2T*>(out2), in_offsets, out_offsets, static_cast<const PermT*>(perm), num_segments, total);
  return launch_status();
}

template <typename ElemT>
int launch_perm_of(const void* in, void* out, const void* in_offsets, const void* out_offsets, const void* perm,
                   int offset_bytes, int perm_bytes, int64_t num_segments, int64_t total, cudaStream_t stream) {
  if (offset_bytes == 8)
    return perm_bytes == 4 ? launch_perm<ElemT, NoElem, int64_t, int32_t, false>(in, out, nullptr, nullptr, in_offsets, out_offsets, perm, num_segments, total, stream)
                           : launch_perm<ElemT, NoElem, int64_t, int64_t, false>(in, out, nullptr, nullptr, in_offsets, out_offsets, perm, num_segments, total, stream);
  return perm_bytes == 4 ? launch_perm<ElemT, NoElem, int32_t, int32_t, false>(in, out, nullptr, nullptr, in_offsets, out_offsets, perm, num_segments, total, stream)
                         : launch_perm<ElemT, NoElem, int32_t, int64_t, false>(in, out, nullptr, nullptr, in_offsets, out_offsets, perm, num_segments, total, stream);
}

// ---- rows of a [T, B] matrix of lengths as segments ------------------------------------------------
// A CTA takes one chunk of one row: of an input row, to sum it; of an output row, to copy its lengths.
constexpr int kLenThreads = 256;
constexpr int kLenItems = 16;
constexpr int kLenChunk = kLenThreads * kLenItems;

template <typename LenT, typename PermT>
__global__ void __launch_bounds__(kLenThreads)
    permute_lengths_kernel(const LenT* __restrict__ lengths, const PermT* __restrict__ perm,
                           LenT* __restrict__ permuted, int64_t* __restrict__ chunk_sums, int64_t rows, int64_t cols,
                           int64_t chunks) {
  __shared__ int64_t warp_sums[kLenThreads / 32];
  const int64_t y = blockIdx.x / chunks, chunk = blockIdx.x - y * chunks;
  const int64_t c0 = chunk * kLenChunk + threadIdx.x;
  int64_t from = y;
  if (y >= rows) {
    from = static_cast<int64_t>(perm[y - rows]);
    assert(from >= 0 && from < rows);
  }
  const LenT* src = lengths + from * cols;
  LenT v[kLenItems];
#pragma unroll
  for (int k = 0; k < kLenItems; ++k) {
    const int64_t c = c0 + k * kLenThreads;
    v[k] = c < cols ? src[c] : LenT(0);
  }
  if (y >= rows) {
    LenT* dst = permuted + (y - rows) * cols;
#pragma unroll
    for (int k = 0; k < kLenItems; ++k) {
      const int64_t c = c0 + k * kLenThreads;
      if (c < cols) dst[c] = v[k];
    }
    return;
  }
  int64_t sum = 0;
#pragma unroll
  for (int k = 0; k < kLenItems; ++k) sum += static_cast<int64_t>(v[k]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(kFullMask, sum, o);
  if ((threadIdx.x & 31) == 0) warp_sums[threadIdx.x >> 5] = sum;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kLenThreads / 32; ++w) sum += warp_sums[w];
    chunk_sums[y * chunks + chunk] = sum;
  }
}

// Short rows: a group of 2^shift lanes, as many as the row has columns (32 at most), takes one. (With a CTA per row
// and one CTA finding all places, below, a call over 20 000 / 100 000 / 1 000 000 rows took 152 / 721 / 7096 us; 52 /
// 54 / 103 now.)
constexpr int kShortCols = 512;

template <typename LenT, typename PermT>
__global__ void __launch_bounds__(kLenThreads)
    permute_short_lengths_kernel(const LenT* __restrict__ lengths, const PermT* __restrict__ perm,
                                 LenT* __restrict__ permuted, int64_t* __restrict__ row_sums, int64_t rows, int cols,
                                 int64_t out_rows, int shift) {
  const int64_t y = (static_cast<int64_t>(blockIdx.x) * kLenThreads + threadIdx.x) >> shift;
  const int g = 1 << shift, lane = threadIdx.x & (g - 1);
  int64_t sum = 0;
  if (y < rows) {
    const LenT* src = lengths + y * cols;
#pragma unroll 4
    for (int c = lane; c < cols; c += g) sum += static_cast<int64_t>(src[c]);
  } else if (y < rows + out_rows) {
    const int64_t from = static_cast<int64_t>(perm[y - rows]);
    assert(from >= 0 && from < rows);
    const LenT* src = lengths + from * cols;
    LenT* dst = permuted + (y - rows) * cols;
#pragma unroll 4
    for (int c = lane; c < cols; c += g) dst[c] = src[c];
  }
  for (int o = g >> 1; o > 0; o >>= 1) sum += __shfl_xor_sync(kFullMask, sum, o);
  if (y < rows && lane == 0) row_sums[y] = sum;
}

constexpr int kRowThreads = 1024;
constexpr int kRowTile = kRowThreads * 4;   // rows of a tile, where there are more rows than threads

// Exclusive sum over the CTA's threads; *total is the CTA's sum.
__device__ __forceinline__ int64_t exclusive_sum(int64_t v, int64_t* total) {
  __shared__ int64_t warp_sums[kRowThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int64_t incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int64_t up = __shfl_up_sync(kFullMask, incl, o);
    if (lane >= o) incl += up;
  }
  if (lane == 31) warp_sums[warp] = incl;
  __syncthreads();
  const int64_t sum = warp_sums[lane];
  int64_t before = lane < warp ? sum : 0, all = sum;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    before += __shfl_xor_sync(kFullMask, before, o);
    all += __shfl_xor_sync(kFullMask, all, o);
  }
  __syncthreads();   // warp_sums may be written again
  *total = all;
  return before + incl - v;
}

// The lengths of input rows, and of output rows with where they come from.
struct InputRows {
  const int64_t* __restrict__ chunk_sums;
  int64_t chunks;
  __device__ __forceinline__ int64_t length(int64_t r, int64_t*) const {
    int64_t len = 0;
#pragma unroll 4
    for (int64_t k = 0; k < chunks; ++k) len += chunk_sums[r * chunks + k];
    return len;
  }
};
struct SummedRows {
  const int64_t* sums;   // (written earlier in the same launch)
  __device__ __forceinline__ int64_t length(int64_t r, int64_t*) const { return sums[r]; }
};
template <typename PermT>
struct OutputRows {
  const PermT* __restrict__ perm;
  const int64_t* in_offsets;   // (written earlier in the same launch, where one CTA does it all)
  int64_t rows;
  __device__ __forceinline__ int64_t length(int64_t j, int64_t* start) const {
    const int64_t from = static_cast<int64_t>(perm[j]);
    if (from < 0 || from >= rows) {
      *start = 0;
      return 0;
    }
    *start = in_offsets[from];
    return in_offsets[from + 1] - *start;
  }
};

// offsets[i], i in the tile [base, base + kRowThreads * kItems) of n rows = carry + the lengths of the tile's rows
// before i; starts, where given, receives the rows' starts. Returns the tile's sum.
template <int kItems, typename Rows>
__device__ __forceinline__ int64_t tile_offsets(const Rows& r, int64_t base, int64_t n, int64_t carry,
                                                int64_t* offsets, int64_t* __restrict__ starts) {
  const int64_t i0 = base + static_cast<int64_t>(threadIdx.x) * kItems;
  int64_t len[kItems], start[kItems], mine = 0;
#pragma unroll
  for (int k = 0; k < kItems; ++k) {
    len[k] = start[k] = 0;
    if (i0 + k < n) len[k] = r.length(i0 + k, &start[k]);
  }
#pragma unroll
  for (int k = 0; k < kItems; ++k) mine += len[k];
  int64_t total;
  int64_t at = carry + exclusive_sum(mine, &total);
#pragma unroll
  for (int k = 0; k < kItems; ++k) {
    if (i0 + k < n) {
      offsets[i0 + k] = at;
      if (starts != nullptr) starts[i0 + k] = start[k];
    }
    at += len[k];
  }
  return total;
}

// One CTA: where every input row starts, then where every output row starts and where it comes from. Rows of
// many chunks are summed first, a warp per row (one row of 16 M lengths: the whole call 322 us with a thread per
// row, 119 so).
constexpr int64_t kManyChunks = 32;

template <typename PermT, int kItems>
__global__ void __launch_bounds__(kRowThreads)
    permute_row_starts_kernel(const int64_t* __restrict__ chunk_sums, const PermT* __restrict__ perm,
                              int64_t* in_offsets, int64_t* __restrict__ in_start, int64_t* __restrict__ out_offsets,
                              int64_t rows, int64_t chunks, int64_t out_rows) {
  const bool many = chunks >= kManyChunks;
  if (many) {
    const int lane = threadIdx.x & 31;
    for (int64_t r = threadIdx.x >> 5; r < rows; r += kRowThreads / 32) {
      int64_t sum = 0;
#pragma unroll 4
      for (int64_t k = lane; k < chunks; k += 32) sum += chunk_sums[r * chunks + k];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(kFullMask, sum, o);
      if (lane == 0) in_offsets[r] = sum;   // a row's sum stays there until its offset takes the place
    }
    __syncthreads();
  }
  int64_t carry = 0;
  for (int64_t base = 0; base < rows; base += kRowThreads * kItems)
    carry += many ? tile_offsets<kItems>(SummedRows{in_offsets}, base, rows, carry, in_offsets, nullptr)
                  : tile_offsets<kItems>(InputRows{chunk_sums, chunks}, base, rows, carry, in_offsets, nullptr);
  if (threadIdx.x == 0) in_offsets[rows] = carry;
  __syncthreads();
  const OutputRows<PermT> out{perm, in_offsets, rows};
  carry = 0;
  for (int64_t base = 0; base < out_rows; base += kRowThreads * kItems)
    carry += tile_offsets<kItems>(out, base, out_rows, carry, out_offsets, in_start);
  if (threadIdx.x == 0) out_offsets[out_rows] = carry;
}

// The same for many rows, a CTA per tile: the tiles' sums (kept in the offset of the tile's first row), their
// prefixes by one CTA, then the offsets.
template <typename Rows>
__global__ void __launch_bounds__(kRowThreads) row_tile_sums_kernel(const Rows r, int64_t n, int64_t* offsets) {
  const int64_t base = static_cast<int64_t>(blockIdx.x) * kRowTile;
  int64_t sum = 0, unused;
#pragma unroll
  for (int k = 0; k < kRowTile / kRowThreads; ++k) {
    const int64_t i = base + k * kRowThreads + threadIdx.x;
    if (i < n) sum += r.length(i, &unused);
  }
  int64_t total;
  exclusive_sum(sum, &total);
  if (threadIdx.x == 0) offsets[base] = total;
}

__global__ void __launch_bounds__(kRowThreads) row_tile_prefixes_kernel(int64_t n, int64_t* offsets) {
  int64_t carry = 0;
  for (int64_t base = 0; base < n; base += int64_t{kRowTile} * kRowThreads) {
    const int64_t i = base + int64_t{kRowTile} * threadIdx.x;
    const int64_t sum = i < n ? offsets[i] : 0;
    int64_t total;
    const int64_t before = exclusive_sum(sum, &total);
    if (i < n) offsets[i] = carry + before;
    carry += total;
  }
  if (threadIdx.x == 0) offsets[n] = carry;
}

template <typename Rows>
__global__ void __launch_bounds__(kRowThreads)
    row_offsets_kernel(const Rows r, int64_t n, int64_t* offsets, int64_t* __restrict__ starts) {
  const int64_t base = static_cast<int64_t>(blockIdx.x) * kRowTile;
  const int64_t carry = offsets[base];
  __syncthreads();   // every thread has it
  tile_offsets<kRowTile / kRowThreads>(r, base, n, carry, offsets, starts);
}

template <typename Rows>
int launch_row_offsets(const Rows& r, int64_t n, int64_t* offsets, int64_t* starts, cudaStream_t stream) {
  const int64_t tiles = (n + kRowTile - 1) / kRowTile;
  if (tiles > 0x7fffffff) return B200TBE_ERR_TOO_LARGE;
  if (tiles > 0) row_tile_sums_kernel<Rows><<<static_cast<unsigned>(tiles), kRowThreads, 0, stream>>>(r, n, offsets);
  row_tile_prefixes_kernel<<<1, kRowThreads, 0, stream>>>(n, offsets);
  if (tiles > 0) row_offsets_kernel<Rows><<<static_cast<unsigned>(tiles), kRowThreads, 0, stream>>>(r, n, offsets, starts);
  return launch_status();
}

// Up to this many rows one CTA does it all: 4096 rows of 64 lengths 50 -> 34 us a call with four rows per thread;
// the six launches of the other way cost more than that below, and less above.
constexpr int64_t kOneCtaRows = 2 * kRowTile;

int64_t length_chunks(int64_t cols) { return cols > 0 ? (cols + kLenChunk - 1) / kLenChunk : 1; }

template <typename LenT, typename PermT>
int launch_row_starts(const void* lengths_, const void* perm_, void* permuted_, int64_t* in_start, int64_t* out_offsets,
                      int64_t rows, int64_t cols, int64_t out_rows, int64_t* scratch, cudaStream_t stream) {
  const LenT* lengths = static_cast<const LenT*>(lengths_);
  const PermT* perm = static_cast<const PermT*>(perm_);
  LenT* permuted = static_cast<LenT*>(permuted_);
  const int64_t chunks = length_chunks(cols);
  const int64_t copied = permuted != nullptr ? out_rows : 0;
  int64_t* in_offsets = scratch;
  int64_t* chunk_sums = scratch + rows + 1;
  if (cols <= kShortCols) {
    int shift = 0;
    while (shift < 5 && (1 << shift) < cols) ++shift;
    const int64_t ctas = (((rows + copied) << shift) + kLenThreads - 1) / kLenThreads;
    if (ctas > 0x7fffffff) return B200TBE_ERR_TOO_LARGE;
    permute_short_lengths_kernel<LenT, PermT><<<static_cast<unsigned>(ctas), kLenThreads, 0, stream>>>(
        lengths, perm, permuted, chunk_sums, rows, static_cast<int>(cols), copied, shift);
  } else {
    const int64_t ctas = (rows + copied) * chunks;
    if (ctas > 0x7fffffff) return B200TBE_ERR_TOO_LARGE;
    permute_lengths_kernel<LenT, PermT><<<static_cast<unsigned>(ctas), kLenThreads, 0, stream>>>(
        lengths, perm, permuted, chunk_sums, rows, cols, chunks);
  }
  if (rows <= kRowThreads && out_rows <= kRowThreads) {
    permute_row_starts_kernel<PermT, 1><<<1, kRowThreads, 0, stream>>>(chunk_sums, perm, in_offsets, in_start,
                                                                       out_offsets, rows, chunks, out_rows);
    return launch_status();
  }
  if (rows <= kOneCtaRows && out_rows <= kOneCtaRows) {
    permute_row_starts_kernel<PermT, 4><<<1, kRowThreads, 0, stream>>>(chunk_sums, perm, in_offsets, in_start,
                                                                       out_offsets, rows, chunks, out_rows);
    return launch_status();
  }
  const int st = launch_row_offsets(InputRows{chunk_sums, chunks}, rows, in_offsets, nullptr, stream);
  if (st != B200TBE_OK) return st;
  return launch_row_offsets(OutputRows<PermT>{perm, in_offsets, rows}, out_rows, out_offsets, in_start, stream);
}

}  // namespace
}  // namespace b200tbe

using namespace b200tbe;

extern "C" int b200tbe_permute_segments(const void* in, void* out, const void* in_offsets,
                                        const void* out_offsets, const void* perm,
                                        int64_t num_segments, int64_t total_elems, int32_t elem_bytes,
                                        int32_t offset_bytes, int32_t perm_bytes,
                                        b200tbe_stream_t stream_) {
  if (num_segments < 0 || total_elems < 0) return B200TBE_ERR_BAD_ARG;
  if (num_segments == 0 || total_elems == 0) return B200TBE_OK;
  if (in == nullptr || out == nullptr || in_offsets == nullptr || out_offsets == nullptr || perm == nullptr)
    return B200TBE_ERR_BAD_ARG;
  if ((offset_bytes != 4 && offset_bytes != 8) || (perm_bytes != 4 && perm_bytes != 8))
    return B200TBE_ERR_BAD_ARG;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  switch (elem_bytes) {
    case 8: return launch_perm_of<uint64_t>(in, out, in_offsets, out_offsets, perm, offset_bytes, perm_bytes, num_segments, total_elems, stream);
    case 4: return launch_perm_of<uint32_t>(in, out, in_offsets, out_offsets, perm, offset_bytes, perm_bytes, num_segments, total_elems, stream);
    case 2: return launch_perm_of<uint16_t>(in, out, in_offsets, out_offsets, perm, offset_bytes, perm_bytes, num_segments, total_elems, stream);
    default: return B200TBE_ERR_UNSUPPORTED;
  }
}

extern "C" size_t b200tbe_permute_row_starts_scratch_bytes(int64_t rows, int64_t cols) {
  if (rows < 0 || cols < 0) return 0;
  return static_cast<size_t>(rows + 1 + rows * length_chunks(cols)) * 8;
}

extern "C" int b200tbe_permute_row_starts(const void* lengths, const void* perm, void* permuted_lengths,
                                          int64_t* in_start, int64_t* out_offsets, int64_t rows, int64_t cols,
                                          int64_t out_rows, int32_t length_bytes, int32_t perm_bytes, void* scratch,
                                          size_t scratch_bytes, b200tbe_stream_t stream_) {
  if (rows < 0 || cols < 0 || out_rows < 0 || (rows == 0 && out_rows > 0)) return B200TBE_ERR_BAD_ARG;
  if ((length_bytes != 4 && length_bytes != 8) || (perm_bytes != 4 && perm_bytes != 8)) return B200TBE_ERR_BAD_ARG;
  if (out_offsets == nullptr || (out_rows > 0 && (in_start == nullptr || perm == nullptr)) ||
      (rows > 0 && cols > 0 && lengths == nullptr))
    return B200TBE_ERR_BAD_ARG;
  if (scratch == nullptr || scratch_bytes < b200tbe_permute_row_starts_scratch_bytes(rows, cols) ||
      !aligned_to(scratch, 8))
    return B200TBE_ERR_SCRATCH;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  if (rows == 0)
    return cudaMemsetAsync(out_offsets, 0, 8, stream) == cudaSuccess ? B200TBE_OK : B200TBE_ERR_LAUNCH;
  int64_t* words = static_cast<int64_t*>(scratch);
  if (length_bytes == 8)
    return perm_bytes == 8 ? launch_row_starts<int64_t, int64_t>(lengths, perm, permuted_lengths, in_start, out_offsets, rows, cols, out_rows, words, stream)
                           : launch_row_starts<int64_t, int32_t>(lengths, perm, permuted_lengths, in_start, out_offsets, rows, cols, out_rows, words, stream);
  return perm_bytes == 8 ? launch_row_starts<int32_t, int64_t>(lengths, perm, permuted_lengths, in_start, out_offsets, rows, cols, out_rows, words, stream)
                         : launch_row_starts<int32_t, int32_t>(lengths, perm, permuted_lengths, in_start, out_offsets, rows, cols, out_rows, words, stream);
}

namespace b200tbe {
namespace {
template <typename ElemT, typename Elem2T>
int move_rows(const void* in, void* out, const void* in2, void* out2, const int64_t* in_start, const int64_t* out_offsets,
              int64_t rows, int64_t total, cudaStream_t stream) {
  return launch_perm<ElemT, Elem2T, int64_t, int32_t, true>(in, out, in2, out2, in_start, out_offsets, nullptr, rows, total,
                                                           stream);
}
}  // namespace
}  // namespace b200tbe

extern "C" int b200tbe_permute_rows(const void* in, void* out, int32_t elem_bytes, const void* in2, void* out2,
                                    int32_t elem2_bytes, const int64_t* in_start, const int64_t* out_offsets,
                                    int64_t out_rows, int64_t total_elems, b200tbe_stream_t stream_) {
  if (out_rows < 0 || total_elems < 0) return B200TBE_ERR_BAD_ARG;
  if (out_rows == 0 || total_elems == 0) return B200TBE_OK;
  if (in == nullptr || out == nullptr || in_start == nullptr || out_offsets == nullptr || (in2 == nullptr) != (out2 == nullptr))
    return B200TBE_ERR_BAD_ARG;
  auto moved = [](int bytes) { return bytes == 2 || bytes == 4 || bytes == 8; };
  if (!moved(elem_bytes) || (in2 != nullptr && !moved(elem2_bytes))) return B200TBE_ERR_UNSUPPORTED;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  const int second = in2 != nullptr ? elem2_bytes : 0;
  switch (elem_bytes * 16 + second) {
    case 8 * 16: return move_rows<uint64_t, NoElem>(in, out, nullptr, nullptr, in_start, out_offsets, out_rows, total_elems, stream);
    case 4 * 16: return move_rows<uint32_t, NoElem>(in, out, nullptr, nullptr, in_start, out_offsets, out_rows, total_elems, stream);
    case 2 * 16: return move_rows<uint16_t, NoElem>(in, out, nullptr, nullptr, in_start, out_offsets, out_rows, total_elems, stream);
    case 8 * 16 + 4: return move_rows<uint64_t, uint32_t>(in, out, in2, out2, in_start, out_offsets, out_rows, total_elems, stream);
    case 4 * 16 + 4: return move_rows<uint32_t, uint32_t>(in, out, in2, out2, in_start, out_offsets, out_rows, total_elems, stream);
    default: break;
  }
  // any other pair of widths: one array after the other
  const int st = b200tbe_permute_rows(in, out, elem_bytes, nullptr, nullptr, 0, in_start, out_offsets, out_rows, total_elems, stream_);
  if (st != B200TBE_OK) return st;
  return b200tbe_permute_rows(in2, out2, second, nullptr, nullptr, 0, in_start, out_offsets, out_rows, total_elems, stream_);
}
