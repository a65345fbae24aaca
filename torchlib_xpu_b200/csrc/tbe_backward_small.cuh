// Plan, linearise and sort of a small batch (at most kSmallSortMax lookups) in one launch.
//
// The general path takes seven launches of 2 to 7 us for this (linearise with the plan, histogram and scatter for
// each of three passes) with gaps between them: 8 tables x 256 samples (11 000 lookups) spend 28 us in its kernels and
// 15 us in this one, a training step 112 and 90 us; 60 000 lookups of two tables 35 us either way, a step 95 and 91.
// One cluster of eight CTAs sorts one table: every CTA holds an eighth of the table's lookups in registers (whatever the
// distribution over the tables, a table's lookups fit a cluster), and per pass of up to 8 bits
//   * ranks its keys by digit, warp by warp (one vote per digit bit, as in radix_sort.cu),
//   * reads the other seven CTAs' digit counts out of their shared memory, and
//   * writes key and payload to their places; the next pass reads them back from L2.
// What bounds it is the chain of those steps (two cluster barriers and two memory round trips per pass);
// the keys are split evenly over the eight CTAs to keep each step short. The result -- the order, the plan,
// the payloads -- is that of the general path.
//
// Part of tbe_backward.cu: included there inside its namespace, after BwdDev and span_for.
#pragma once

constexpr int kSmallThreads = 512;
constexpr int kSmallWarps = kSmallThreads / 32;
constexpr int kSmallItems = 16;                                       // keys per thread
constexpr int kSmallCluster = 8;                                      // CTAs per table
constexpr int kSmallSortMax = kSmallCluster * kSmallThreads * kSmallItems;   // 65536
// A table takes a cluster however few lookups it has, and some 37 clusters run at a time: training steps of 41 000
// lookups over 32 / 64 / 80 / 96 / 112 / 128 tables take 91 / 82 / 86 / 92 / 104 / 109 us this way (the kernel 14 / 26 /
// - / - / - / 49) and 101 / 94 / 95 / 95 / 93 / 94 by the general path.
constexpr int kSmallSortTables = 96;
constexpr int kSmallRadix = 256;
constexpr int kSmallBags = 4096;                                      // bag starts kept in shared memory

struct SmallSort {
  uint32_t* keys[2];      // pass 0 writes [0], pass 1 [1], ...
  uint32_t* vals[2];
  uint32_t* seg_start;    // the plan, as build_sort_plan writes it
  uint32_t* total_tiles;
  uint4* tile_desc;
  int32_t max_tiles;
  int32_t key_bits;
};

template <typename IndexT, bool kWeighted>
__global__ void __cluster_dims__(kSmallCluster, 1, 1) __launch_bounds__(kSmallThreads, 2)
    small_sort_kernel(const __grid_constant__ BwdDev p, const __grid_constant__ SmallSort s) {
  __shared__ uint16_t warp_hist[kSmallWarps][kSmallRadix];
  __shared__ uint32_t cta_hist[kSmallRadix];     // read by the other CTAs of the cluster
  __shared__ uint32_t digit_pos[kSmallRadix];
  __shared__ uint32_t bag_start[kSmallBags];
  cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  const int rank_in_cluster = static_cast<int>(cluster.block_rank());
  const int t = static_cast<int>(blockIdx.x) / kSmallCluster;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t lanemask_lt = (1u << lane) - 1u;
  const int64_t n = p.num_indices;

  auto start_of = [&](int seg) -> uint32_t {
    int64_t v = load_index<IndexT>(p.offsets, static_cast<int64_t>(seg) * p.B);
    if (v < 0) v = 0;
    return static_cast<uint32_t>(v > n ? n : v);
  };
  const uint32_t seg_begin = start_of(t);
  const uint32_t seg_next = start_of(t + 1);
  const uint32_t seg_len = seg_next > seg_begin ? seg_next - seg_begin : 0u;

  // ---- the plan: this table's tiles follow those of the tables before it ----
  if (rank_in_cluster == 0) {
    uint32_t before = 0;
    bool ordered = seg_begin <= seg_next;
    for (int q = threadIdx.x; q < t; q += kSmallThreads) {
      const uint32_t a = start_of(q), b = start_of(q + 1);
      before += b > a ? (b - a + kSortPlanTile - 1) / kSortPlanTile : 0u;
      ordered = ordered && a <= b;
    }
    const bool good = __syncthreads_and(ordered);   // of the tables up to this one: the last table's CTA sees all
    uint32_t first;
    block_exclusive_scan(before, &first);
    const uint32_t tiles = (seg_len + kSortPlanTile - 1) / kSortPlanTile;
    for (uint32_t q = threadIdx.x; q < tiles; q += kSmallThreads) {
      const uint32_t done = q * kSortPlanTile;
      const uint32_t count = seg_len - done < static_cast<uint32_t>(kSortPlanTile) ? seg_len - done : kSortPlanTile;
      if (first + q < static_cast<uint32_t>(s.max_tiles))
        s.tile_desc[first + q] = make_uint4(seg_begin + done, count, static_cast<uint32_t>(t), first);
    }
    if (threadIdx.x == 0) {
      s.seg_start[t] = seg_begin;
      if (t == p.T - 1) {
        s.seg_start[p.T] = seg_next;
        // tables that end before they begin would overlap others: nothing is done with what is sorted
        if (!good && p.status != nullptr) atomicOr(p.status, B200TBE_DEV_OFFSETS_NOT_MONOTONE);
        *s.total_tiles = good ? first + tiles : 0u;
      }
    }
  }

  if (seg_len == 0) return;   // the whole cluster

  // ---- this CTA's lookups: an eighth of the table's, in order ----
  const uint32_t each = (seg_len + kSmallCluster - 1) / kSmallCluster;
  const uint32_t c_begin = each * rank_in_cluster < seg_len ? each * rank_in_cluster : seg_len;
  const int c_n = static_cast<int>(seg_len - c_begin < each ? seg_len - c_begin : each);
  // keys per thread, and the warp's share: item r of lane l of warp w is lookup w * items * 32 + r * 32 + l
  const int items = static_cast<int>((each + kSmallThreads - 1) / kSmallThreads);
  const int warp_base = warp * items * 32;

  // ---- linearise: key = row id, payload = bag (or position, when weights travel along) ----
  const bool bags_here = p.B <= kSmallBags;
  const int64_t bag0 = static_cast<int64_t>(t) * p.B;
  if (bags_here)
    for (int b = threadIdx.x; b < p.B; b += kSmallThreads) {
      const int64_t v = load_index<IndexT>(p.offsets, bag0 + b);
      bag_start[b] = v < 0 ? 0u : (v > n ? static_cast<uint32_t>(n) : static_cast<uint32_t>(v));
    }
  uint32_t k[kSmallItems], v[kSmallItems];
  int64_t rows = __ldg(p.hash_size_cumsum + t + 1) - __ldg(p.hash_size_cumsum + t);
  const int64_t sortable = int64_t{1} << s.key_bits;
  if (rows > sortable) {   // the caller's bound on rows per table was too small for this table
    if (p.status != nullptr) atomicOr(p.status, B200TBE_DEV_UNSUPPORTED_SHAPE);
    rows = sortable;
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kSmallItems; ++r) {
    k[r] = 0;
    v[r] = kInvalidPayload;
    const int it = warp_base + r * 32 + lane;
    if (r >= items || it >= c_n) continue;
    const uint32_t j = seg_begin + c_begin + it;
    const int64_t idx = load_index<IndexT>(p.indices, j);
    // the last bag of the table that starts at or before j
    int lo = 0, hi = p.B - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      const int64_t start = bags_here ? static_cast<int64_t>(bag_start[mid]) : load_index<IndexT>(p.offsets, bag0 + mid);
      if (start <= static_cast<int64_t>(j)) {
        lo = mid;
      } else {
        hi = mid - 1;
      }
    }
    const uint32_t bag = static_cast<uint32_t>(bag0 + lo);
    if (kWeighted) p.bag_of_pos[j] = bag;
    if (idx < 0 || idx >= rows) {
      if (p.status != nullptr) atomicOr(p.status, B200TBE_DEV_INDEX_OUT_OF_RANGE);
    } else {
      k[r] = static_cast<uint32_t>(idx);
      v[r] = kWeighted ? j : bag;
    }
  }

  // ---- passes ----
  const int passes = (s.key_bits + 7) / 8;
  int shift = 0;
  for (int pass = 0; pass < passes; ++pass) {
    const int bits = (s.key_bits - shift + (passes - pass) - 1) / (passes - pass);   // spread evenly
    const uint32_t mask = (1u << bits) - 1u;
    uint32_t* keys_out = s.keys[pass & 1];
    uint32_t* vals_out = s.vals[pass & 1];
    {
      uint32_t* z = reinterpret_cast<uint32_t*>(&warp_hist[0][0]);
      for (int i = threadIdx.x; i < kSmallWarps * kSmallRadix / 2; i += kSmallThreads) z[i] = 0;
    }
    __syncthreads();
    uint32_t rank[kSmallItems / 2];   // two to a register: 64 registers a thread, two CTAs per SM
#pragma unroll
    for (int r = 0; r < kSmallItems; ++r) {
      if (r >= items) break;
      const bool valid = warp_base + r * 32 + lane < c_n;
      const uint32_t d = (k[r] >> shift) & mask;
      uint32_t peers = __ballot_sync(kFullMask, valid);
#pragma unroll
      for (int b = 0; b < 8; ++b) {
        const bool bit = (d >> b) & 1u;
        const uint32_t with_bit = __ballot_sync(kFullMask, bit);
        peers &= bit ? with_bit : ~with_bit;
      }
      const uint32_t before = warp_hist[warp][d];
      const uint32_t my_rank = before + __popc(peers & lanemask_lt);   // < 32 * kSmallItems
      rank[r / 2] = r & 1 ? rank[r / 2] | (my_rank << 16) : my_rank;
      __syncwarp();
      if (valid && (peers & lanemask_lt) == 0) warp_hist[warp][d] = static_cast<uint16_t>(before + __popc(peers));
      __syncwarp();
    }
    __syncthreads();
    // per digit: exclusive prefix over the warps, the CTA's total
    if (threadIdx.x < kSmallRadix) {
      uint32_t run = 0;
#pragma unroll
      for (int w = 0; w < kSmallWarps; ++w) {
        const uint32_t c = warp_hist[w][threadIdx.x];
        warp_hist[w][threadIdx.x] = static_cast<uint16_t>(run);
        run += c;
      }
      cta_hist[threadIdx.x] = run;
    }
    cluster.sync();
    // over the cluster: keys of this digit in the CTAs before this one, and in all of them
    uint32_t before = 0, all = 0;
    if (threadIdx.x < kSmallRadix) {
      uint32_t c[kSmallCluster];
#pragma unroll
      for (int q = 0; q < kSmallCluster; ++q) c[q] = *cluster.map_shared_rank(&cta_hist[threadIdx.x], q);
#pragma unroll
      for (int q = 0; q < kSmallCluster; ++q) {
        if (q < rank_in_cluster) before += c[q];
        all += c[q];
      }
    }
    uint32_t unused_total;
    const uint32_t start = block_exclusive_scan(all, &unused_total);
    if (threadIdx.x < kSmallRadix) digit_pos[threadIdx.x] = seg_begin + start + before;
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kSmallItems; ++r) {
      if (r >= items) break;
      if (warp_base + r * 32 + lane < c_n) {
        const uint32_t d = (k[r] >> shift) & mask;
        const uint32_t pos = digit_pos[d] + warp_hist[warp][d] + (r & 1 ? rank[r / 2] >> 16 : rank[r / 2] & 0xffffu);
        keys_out[pos] = k[r];
        vals_out[pos] = v[r];
      }
    }
    // the cluster's keys are in place before any of its CTAs reads them, and its counts have been read
    // before any of them is written again
    __threadfence();
    cluster.sync();
    shift += bits;
    if (pass + 1 < passes) {
#pragma unroll
      for (int r = 0; r < kSmallItems; ++r) {
        const int it = warp_base + r * 32 + lane;
        if (r >= items || it >= c_n) continue;
        k[r] = __ldcg(keys_out + seg_begin + c_begin + it);
        v[r] = __ldcg(vals_out + seg_begin + c_begin + it);
      }
    }
  }
}

// Launches the sort; *result is the buffer (0 or 1) the sorted pairs end in.
template <typename IndexT>
int launch_small_sort(const BwdDev& d, const SmallSort& s, bool weighted, int* result, cudaStream_t stream) {
  const int64_t ctas = static_cast<int64_t>(d.T) * kSmallCluster;
  if (ctas > 0x7fffffff) return B200TBE_ERR_TOO_LARGE;
  if (weighted) {
    small_sort_kernel<IndexT, true><<<static_cast<unsigned>(ctas), kSmallThreads, 0, stream>>>(d, s);
  } else {
    small_sort_kernel<IndexT, false><<<static_cast<unsigned>(ctas), kSmallThreads, 0, stream>>>(d, s);
  }
  *result = ((s.key_bits + 7) / 8 - 1) & 1;
  return launch_status();
}
