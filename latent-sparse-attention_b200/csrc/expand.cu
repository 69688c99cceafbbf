// Expansion: a row's picked buckets become its read list - members best bucket first, then the window, then
// the sinks. Pure integer work, one warp a row, ballot-compacted so the order is the table's order.
#include "common.cuh"
#include "expand.cuh"

namespace lsa {

constexpr int kExpandWarps = 8;
constexpr int kFlatCap = 64, kFlatChunks = 8;

struct ExpandParams {
  const int32_t *picked;      // [R, top_p]
  const int64_t *positions;   // [R]
  const int32_t *members;     // [m, cap]
  const int32_t *row_top_p;   // [R] or NULL
  const int32_t *row_top_k;   // [R] or NULL
  const int32_t *page_table;  // [pages] (or [requests, pages] with page_table_stride) or NULL
  const int32_t *row_request;   // [R] request of each row, or NULL for request 0
  const int32_t *bucket_pages;  // [requests, bucket_max_pages] page of every bucket_page_rows logical buckets, or NULL
  int64_t page_table_stride, bucket_pages_stride;
  int bucket_page_rows, bucket_max_pages;
  int32_t *selected;          // [R, width]
  int32_t *lengths;           // [R]
  int32_t *status;
  int64_t R, m, owner_first, owner_end;
  int top_p, cap, top_k, sink, window, page_size, width, granule, world, rank, flags;
  const int64_t *keys;   // in place of the picks: `parts` lists a row of sorted keys [parts, R, top_p] (expand_spread_kernel's SORTED)
  int parts, size;       // (size: top_p as the next power of two)
  uint32_t cap_inverse;  // ceil(2^21 / cap)
  bool keeps_all;        // no owner range and no dealt granules: every id is kept
};

// A row's own budget, or the call's. (A row with less than nothing to spend, or before position 0, has an empty list.)
__device__ __forceinline__ int budget(const int32_t *rows, int64_t r, int most) {
  return rows ? max(0, min(rows[r], most)) : most;
}

// Whether this caller keeps an id: inside its contiguous range and, when the cache is dealt out in granules of
// positions round-robin over `world` ranks, in one of its granules.
__device__ __forceinline__ bool owned(const ExpandParams &p, int64_t id) {
  if (id < p.owner_first || id >= p.owner_end) return false;
  if (p.world <= 1) return true;
  const uint32_t u = (uint32_t)id;  // (an id fits 31 bits - the lists are int32 - and 32-bit division is the cheap one)
  return (int)((u / (uint32_t)p.granule) % (uint32_t)p.world) == p.rank;
}

// What is written for an id: the position, its row in the rank's own cache when granules are dealt out, or its KV
// slot through the page table.
__device__ __forceinline__ int32_t stored_id(const ExpandParams &p, const int32_t *table, int64_t id) {
  uint32_t u = (uint32_t)id;
  if (p.world > 1) u = u / ((uint32_t)p.granule * (uint32_t)p.world) * (uint32_t)p.granule + u % (uint32_t)p.granule;
  if (!table) return (int32_t)u;
  return table[u / (uint32_t)p.page_size] * p.page_size + (int32_t)(u % (uint32_t)p.page_size);
}

// Append the owned ids of [first, end) to out[written..], in order; returns the new count.
__device__ __forceinline__ int append_run(const ExpandParams &p, const int32_t *table, int32_t *out, int written,
                                          int64_t first, int64_t end, int lane) {
  const unsigned below = (1u << lane) - 1;
  for (int64_t base = first; base < end; base += 32) {
    const int64_t t = base + lane;
    const bool mine = t < end && owned(p, t);
    const unsigned keeps = __ballot_sync(0xffffffffu, mine);
    if (mine) out[written + __popc(keeps & below)] = stored_id(p, table, t);
    written += __popc(keeps);
  }
  return written;
}

__global__ void __launch_bounds__(kExpandWarps * 32) expand_kernel(ExpandParams p) {
  const int lane = lane_id();
  const int64_t r = (int64_t)blockIdx.x * kExpandWarps + (threadIdx.x >> 5);
  dependents_may_launch();
  wait_for_earlier_grids();
  if (r >= p.R) return;
  const int64_t pos = p.positions[r];
  const int64_t request = p.row_request ? p.row_request[r] : 0;
  const int32_t *table = p.page_table ? p.page_table + request * p.page_table_stride : nullptr;
  const int row_p = budget(p.row_top_p, r, p.top_p), row_k = budget(p.row_top_k, r, p.top_k);
  const int64_t window_start = max((int64_t)0, pos + 1 - p.window);
  int32_t *out = p.selected + r * p.width;
  const unsigned below = (1u << lane) - 1;
  int counted = 0;  // ids that count toward top_k
  int written = 0;  // ids this owner keeps
  int bad = 0;
  // The picks are read 32 at a time, a lane a pick (so no load waits on the one before), and a bucket's member
  // chunks four at a time: the loads of a group are in flight together, only the counting is in order. A bucket's
  // members ascend and its row ends in padding, so the first chunk that holds padding or a member inside the window
  // is the last one of the bucket that can count: the rest of its row (half of it, on average) is never read.
  for (int i0 = 0; i0 < row_p && counted < row_k; i0 += 32) {
    int64_t my_bucket = -1;
    if (i0 + lane < row_p) {
      my_bucket = p.picked[r * p.top_p + i0 + lane];
      if (my_bucket >= 0 && p.bucket_pages) {
        // a request's logical bucket sits at row bucket % rows of its page bucket / rows
        const int64_t slot = my_bucket / p.bucket_page_rows;
        const int page = slot < p.bucket_max_pages ? p.bucket_pages[request * p.bucket_pages_stride + slot] : -1;
        my_bucket = page >= 0 ? (int64_t)page * p.bucket_page_rows + my_bucket % p.bucket_page_rows : p.m;
      }
      if (my_bucket >= p.m) {
        my_bucket = -1;
        ++bad;
      }
    }
    const int picks = min(32, row_p - i0);
    // Buckets of at most 64 members: the picks' rows one after another as ONE walk, 256 places a step, so that a step of
    // eight loads and ballots serves 256 / cap picks and not one of them. (What bounds it is the warp's own instructions:
    // 7,613 rows of 1,024 picks of 16 took 1,037 us a pick at a time, and take 424.)
    if (p.cap <= kFlatCap) {
      const int places = picks * p.cap;
      for (int at0 = 0; at0 < places && counted < row_k; at0 += 32 * kFlatChunks) {
        int32_t ids[kFlatChunks];
#pragma unroll
        for (int j = 0; j < kFlatChunks; ++j) {
          const int at = at0 + 32 * j + lane;
          const int pick = (int)(((uint32_t)at * p.cap_inverse) >> 21);  // at / cap: exact below 32 caps, rounded up to a step
          const int64_t bucket = __shfl_sync(0xffffffffu, my_bucket, pick & 31);
          ids[j] = at < places && bucket >= 0 ? p.members[bucket * p.cap + (at - pick * p.cap)] : LSA_PAD;
        }
#pragma unroll
        for (int j = 0; j < kFlatChunks; ++j) {
          const int32_t id = ids[j];
          const bool counts = id >= p.sink && id < window_start;
          const unsigned votes = __ballot_sync(0xffffffffu, counts);
          const bool inside = counts && counted + __popc(votes & below) < row_k;
          const bool mine = inside && (p.keeps_all || owned(p, id));
          const unsigned keeps = __ballot_sync(0xffffffffu, mine);
          if (mine) out[written + __popc(keeps & below)] = stored_id(p, table, id);
          written += __popc(keeps);
          counted += __popc(votes);
        }
      }
      continue;
    }
    for (int pick = 0; pick < picks && counted < row_k; ++pick) {
      const int64_t bucket = __shfl_sync(0xffffffffu, my_bucket, pick);
      if (bucket < 0) continue;
      const int32_t *row = p.members + bucket * p.cap;
      bool ended = false;
      for (int at0 = 0; at0 < p.cap && !ended && counted < row_k; at0 += 128) {
        int32_t ids[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int at = at0 + 32 * j + lane;
          ids[j] = at < p.cap ? row[at] : LSA_PAD;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int32_t id = ids[j];
          const bool counts = id >= p.sink && id < window_start;
          const unsigned votes = __ballot_sync(0xffffffffu, counts);
          const bool inside = counts && counted + __popc(votes & below) < row_k;
          const bool mine = inside && owned(p, id);
          const unsigned keeps = __ballot_sync(0xffffffffu, mine);
          if (mine) out[written + __popc(keeps & below)] = stored_id(p, table, id);
          written += __popc(keeps);
          counted += __popc(votes);
          ended |= __any_sync(0xffffffffu, id < 0 || id >= window_start);
        }
      }
    }
  }
  bad = warp_sum_int(bad);
  // The window, ascending, then the sinks.
  if (!(p.flags & LSA_EXPAND_NO_LOCAL)) {
    written = append_run(p, table, out, written, window_start, pos + 1, lane);
    written = append_run(p, table, out, written, 0, min((int64_t)p.sink, min(window_start, pos + 1)), lane);
  }
  if (!(p.flags & LSA_EXPAND_NO_PAD))
    for (int j = written + lane; j < p.width; j += 32) out[j] = LSA_PAD;
  if (lane == 0) {
    p.lengths[r] = written;
    if (bad && p.status) atomicAdd(p.status, bad);
  }
}

// Many rows with long lists (a prefill chunk over wide buckets): a CTA of 256 threads a row. Members ascend, so what a
// pick adds to the list is ONE RUN of its row: a thread a pick finds the run's ends by bisection, the counts are scanned
// into offsets, and a warp copies a pick's run eight loads at a time, with no vote on any of its ids. The kernel above
// takes a warp a row, which walks 48,000 ids of a row of the 10M-token MLA context one group of four loads at a time:
// rows of 777 leave most of an SM's warps empty that way, and 8,192 rows wait on one another's votes. Only for callers
// that keep every id, so the ids that count toward top_k are the ids written.
constexpr int kRunThreads = 256;
constexpr int kRunMaxPicks = 1024;
constexpr int kRunAhead = 8;

__global__ void __launch_bounds__(kRunThreads) expand_run_kernel(ExpandParams p) {
  __shared__ int64_t from_s[kRunMaxPicks];  // where the pick's run starts in the member table
  __shared__ int start_s[kRunMaxPicks];     // and in the list
  __shared__ int count_s[kRunMaxPicks];
  __shared__ int warp_total_s[kRunThreads / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int kWarps = kRunThreads / 32;
  const int64_t r = blockIdx.x;
  const int64_t pos = p.positions[r];
  const int64_t request = p.row_request ? p.row_request[r] : 0;
  const int32_t *table = p.page_table ? p.page_table + request * p.page_table_stride : nullptr;
  const int row_p = budget(p.row_top_p, r, p.top_p), row_k = budget(p.row_top_k, r, p.top_k);
  const int64_t window_start = max((int64_t)0, pos + 1 - p.window);
  int32_t *out = p.selected + r * p.width;
  int all = 0, bad = 0;
  for (int i0 = 0; i0 < row_p; i0 += kRunThreads) {
    const int i = i0 + tid;
    int64_t bucket = i < row_p ? p.picked[r * p.top_p + i] : -1;
    if (bucket >= 0 && p.bucket_pages) {
      const int64_t slot = bucket / p.bucket_page_rows;
      const int page = slot < p.bucket_max_pages ? p.bucket_pages[request * p.bucket_pages_stride + slot] : -1;
      bucket = page >= 0 ? (int64_t)page * p.bucket_page_rows + bucket % p.bucket_page_rows : p.m;
    }
    const bool outside = bucket >= p.m;
    if (outside) bucket = -1;
    int first = 0, end = 0;
    if (bucket >= 0) {
      const int32_t *row = p.members + bucket * p.cap;
      int lo = 0, hi = p.cap;  // the first place that is padding or inside the window
      while (lo < hi) {
        const int mid = (lo + hi) >> 1, id = row[mid];
        if (id < 0 || id >= window_start) hi = mid; else lo = mid + 1;
      }
      end = lo;
      while (first < end && row[first] < p.sink) ++first;
    }
    const int n = end - first;
    int incl = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += up;
    }
    if (lane == 31) warp_total_s[warp] = incl;
    __syncthreads();
    int before = all;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      if (w < warp) before += warp_total_s[w];
      all += warp_total_s[w];
    }
    if (i < row_p) {
      const int start = before + incl - n;
      from_s[i] = bucket >= 0 ? bucket * p.cap + first : 0;
      start_s[i] = start;
      count_s[i] = max(0, min(n, row_k - start));
      bad += outside && start < row_k;
    }
    __syncthreads();
  }
  for (int pick = warp; pick < row_p; pick += kWarps) {
    const int n = count_s[pick];
    const int32_t *src = p.members + from_s[pick];
    int32_t *dst = out + start_s[pick];
    for (int at0 = 0; at0 < n; at0 += 32 * kRunAhead) {
      int32_t ids[kRunAhead];
#pragma unroll
      for (int j = 0; j < kRunAhead; ++j) {
        const int at = at0 + 32 * j + lane;
        ids[j] = at < n ? src[at] : 0;
      }
#pragma unroll
      for (int j = 0; j < kRunAhead; ++j) {
        const int at = at0 + 32 * j + lane;
        if (at < n) dst[at] = table ? stored_id(p, table, ids[j]) : ids[j];
      }
    }
  }
  int total = min(all, row_k);
  if (!(p.flags & LSA_EXPAND_NO_LOCAL)) {
    const int in_window = (int)max((int64_t)0, pos + 1 - window_start);
    for (int i = tid; i < in_window; i += kRunThreads) out[total + i] = stored_id(p, table, window_start + i);
    total += in_window;
    const int sinks = (int)max((int64_t)0, min((int64_t)p.sink, min(window_start, pos + 1)));
    for (int i = tid; i < sinks; i += kRunThreads) out[total + i] = stored_id(p, table, i);
    total += sinks;
  }
  if (!(p.flags & LSA_EXPAND_NO_PAD))
    for (int j = total + tid; j < p.width; j += kRunThreads) out[j] = LSA_PAD;
  if (tid == 0) p.lengths[r] = total;
  bad = warp_sum_int(bad);
  if (lane == 0 && bad && p.status) atomicAdd(p.status, bad);
}

// A few rows with long lists (a decode step): `gridDim.x` CTAs a row. Members ascend, so how many of a pick count is found
// without reading its row: a warp looks at 32 places spread over it and then at the places between two of them, two rounds of
// loads for every pick at once. Every CTA finds all picks' counts and scans them - the same few loads, and nothing to exchange
// - and writes its share of the list, a thread an id: the pick that owns it by bisection of the scanned counts. Only for
// callers that keep every id, so the ids that count toward top_k are the ids written. What bounds it is four dependent rounds
// of loads (positions and picks, the two of the counts, the ids). (A row of 83,000 ids from 128 picks of up to 1,280: 10.5 us in a
// cluster of eight CTAs whose warps read a whole bucket each to count it, 9.6 this way, and in a decode step, where the members
// come out of HBM, 15.6 and 9.6; 3,100 ids from 64 picks of 64 5.9 and 5.7, 64 rows of 9,200 from 32 picks of 512 7.6 and 6.9 in
// a CTA a row that did the same.)
constexpr int kSpreadThreads = 1024;
constexpr int kSpreadMaxPicks = 1024;
constexpr int kSpreadMaxCtas = 32;
constexpr int kSpreadPicks = 4;  // picks a warp looks at side by side

// SORTED: the picks are the best of several lists, placed by counting as in a merge of its own - every CTA all of them, a thread a
// key. (128 picks of 16,384 buckets out of the lists of eight clusters, a row of 83,000 ids: the merge 6.2 and the expansion 9.3 us as
// two launches, 13.6 as one; the decode step over 10M positions 68.5 -> 66.3.)
constexpr int kSortedParts = 8, kSortedPicks = 128;

template <bool SORTED>
__global__ void __launch_bounds__(kSpreadThreads) expand_spread_kernel(ExpandParams p) {
  __shared__ int64_t from_s[kSpreadMaxPicks];  // where the pick's run starts in the member table
  __shared__ int count_s[kSpreadMaxPicks];
  __shared__ int start_s[kSpreadMaxPicks + 1];  // and in the list
  __shared__ int bad_s;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int kWarps = kSpreadThreads / 32;
  const int64_t r = blockIdx.y;
  dependents_may_launch();
  wait_for_earlier_grids();
  const int64_t pos = p.positions[r];
  const int64_t request = p.row_request ? p.row_request[r] : 0;
  const int32_t *table = p.page_table ? p.page_table + request * p.page_table_stride : nullptr;
  const int row_p = budget(p.row_top_p, r, p.top_p), row_k = budget(p.row_top_k, r, p.top_k);
  const int64_t window_start = max((int64_t)0, pos + 1 - p.window);
  int32_t *out = p.selected + r * p.width;
  if (tid == 0) bad_s = 0;
  __shared__ int64_t keys_s[SORTED ? kSortedParts * kSortedPicks : 1];
  __shared__ int32_t pick_s[SORTED ? kSortedPicks : 1];
  if constexpr (SORTED) {
    static_assert(kSortedParts * kSortedPicks <= kSpreadThreads, "a thread a key");
    if (tid < p.parts * p.size) {
      const int part = tid / p.size, i = tid - part * p.size;
      keys_s[tid] = i < p.top_p ? p.keys[((int64_t)part * p.R + r) * p.top_p + i] : kEmptyKey;
    }
    if (tid < p.top_p) pick_s[tid] = LSA_PAD;
    __syncthreads();
    // (at least top_p keys reach the least of the lists' keys at place ceil(top_p / parts))
    const int deep = (p.top_p + p.parts - 1) / p.parts - 1;
    int64_t least = INT64_MAX;
    for (int j = 0; j < p.parts; ++j) least = min(least, keys_s[j * p.size + deep]);
    const int i = tid / p.parts, part = tid - i * p.parts;  // (the lists' heads first: what is under the bar is whole warps)
    const int64_t key = i < p.top_p ? keys_s[part * p.size + i] : kEmptyKey;
    if (key >= least && key != kEmptyKey) {
      int rank = i;
#pragma unroll 4
      for (int j = 0; j < p.parts; ++j) {
        const int before = keys_before(keys_s + j * p.size, p.size, key, j < part);
        rank += j == part ? 0 : before;
      }
      if (rank < p.top_p) pick_s[rank] = key_id(key);
    }
  }
  __syncthreads();
  for (int i = tid; i < row_p; i += kSpreadThreads) {
    int64_t bucket = SORTED ? pick_s[i] : p.picked[r * p.top_p + i];
    if (bucket >= 0 && p.bucket_pages) {
      const int64_t slot = bucket / p.bucket_page_rows;
      const int page = slot < p.bucket_max_pages ? p.bucket_pages[request * p.bucket_pages_stride + slot] : -1;
      bucket = page >= 0 ? (int64_t)page * p.bucket_page_rows + bucket % p.bucket_page_rows : p.m;
    }
    if (bucket >= p.m) {
      bucket = -1;
      atomicAdd(&bad_s, 1);
    }
    from_s[i] = bucket >= 0 ? bucket * p.cap : -1;
  }
  __syncthreads();
  for (int i0 = warp * kSpreadPicks; i0 < row_p; i0 += kWarps * kSpreadPicks) {
    int64_t at[kSpreadPicks];
    int first[kSpreadPicks], count[kSpreadPicks];
#pragma unroll
    for (int j = 0; j < kSpreadPicks; ++j) at[j] = i0 + j < row_p ? from_s[i0 + j] : -1;
    member_runs(p.members, p.cap, at, window_start, p.sink, first, count);
#pragma unroll
    for (int j = 0; j < kSpreadPicks; ++j)
      if (lane == 0 && i0 + j < row_p) {
        count_s[i0 + j] = count[j];
        if (at[j] >= 0) from_s[i0 + j] = at[j] + first[j];
      }
  }
  __syncthreads();
  if (warp == 0) run_starts(count_s, row_p, start_s);
  __syncthreads();
  const int listed = min(start_s[row_p], row_k);
  const int in_window = p.flags & LSA_EXPAND_NO_LOCAL ? 0 : (int)max((int64_t)0, pos + 1 - window_start);
  const int sinks = p.flags & LSA_EXPAND_NO_LOCAL ? 0 : (int)max((int64_t)0, min((int64_t)p.sink, min(window_start, pos + 1)));
  const int total = listed + in_window + sinks;
  const int gtid = blockIdx.x * kSpreadThreads + tid, gthreads = gridDim.x * kSpreadThreads;
  list_members(p.members, from_s, start_s, row_p, listed, gtid, gthreads, [&](int e, int32_t id) { out[e] = stored_id(p, table, id); });
  for (int i = gtid; i < in_window; i += gthreads) out[listed + i] = stored_id(p, table, window_start + i);
  for (int i = gtid; i < sinks; i += gthreads) out[listed + in_window + i] = stored_id(p, table, i);
  if (!(p.flags & LSA_EXPAND_NO_PAD))
    for (int j = total + gtid; j < p.width; j += gthreads) out[j] = LSA_PAD;
  if (tid == 0 && blockIdx.x == 0) {
    p.lengths[r] = total;
    if (bad_s && p.status) atomicAdd(p.status, bad_s);
  }
}

bool expands_spread(int64_t R, int top_p, int cap, int window) {
  return top_p <= kSpreadMaxPicks && (int64_t)top_p * cap + window >= (R <= 8 ? 1024 : (R <= 64 ? 4096 : INT64_MAX));
}

// As many CTAs a row as give a thread two ids of half-full buckets, a wave of them at most.
static int launch_spread(const ExpandParams &p, cudaStream_t stream) {
  const int64_t wanted = ((int64_t)p.top_p * p.cap / 2 + p.window) / (2 * kSpreadThreads);
  const int64_t most = sm_count() / p.R < kSpreadMaxCtas ? sm_count() / p.R : kSpreadMaxCtas;
  const int64_t ctas = wanted < most ? wanted : most;
  const dim3 grid((unsigned)(ctas < 1 ? 1 : ctas), (unsigned)p.R);
  launch(p.R <= kChainedRows, p.keys ? expand_spread_kernel<true> : expand_spread_kernel<false>, grid, dim3(kSpreadThreads), 0, stream,
         p);
  LSA_LAUNCH_CHECK();
  return LSA_OK;
}

int expand_sorted(const int64_t *keys, int parts, int64_t R, int top_p, const int64_t *positions, int64_t m, const RowLists &to,
                  cudaStream_t stream) {
  LSA_REQUIRE(parts <= kSortedParts && top_p <= kSortedPicks, LSA_ERR_UNSUPPORTED);
  ExpandParams p = {};
  p.keys = keys, p.parts = parts, p.size = 2;
  while (p.size < top_p) p.size <<= 1;
  p.positions = positions, p.members = to.members, p.selected = to.lists, p.lengths = to.lengths;
  p.R = R, p.m = m, p.owner_end = INT64_MAX, p.world = p.granule = 1, p.keeps_all = true;
  p.top_p = top_p, p.cap = to.cap, p.top_k = to.top_k, p.sink = to.sink, p.window = to.window, p.width = (int)to.width;
  p.flags = LSA_EXPAND_NO_PAD;
  return launch_spread(p, stream);
}

}  // namespace lsa

LSA_API int lsa_expand_batched(const int32_t *picked, int64_t R, int top_p, const int64_t *positions,
                       const int32_t *members, int64_t m, int bucket_cap, const int32_t *row_top_p,
                       const int32_t *row_top_k, int top_k, int sink, int window, const int32_t *page_table,
                       int page_size, int64_t owner_first, int64_t owner_end, int owner_granule, int owner_world,
                       int owner_rank, int flags, const int32_t *row_request, int64_t page_table_stride,
                       const int32_t *bucket_pages, int64_t bucket_pages_stride, int bucket_max_pages,
                       int bucket_page_rows, int32_t *selected, int32_t *lengths,
                       int32_t *status, void *stream) {
  LSA_REQUIRE(picked && positions && selected && lengths, LSA_ERR_NULL);
  LSA_REQUIRE(m == 0 || members, LSA_ERR_NULL);
  LSA_REQUIRE(R >= 0 && top_p >= 1 && m >= 0 && bucket_cap >= 1 && top_k >= 1 && sink >= 0 && window >= 1,
              LSA_ERR_ARGUMENT);
  LSA_REQUIRE(!page_table || page_size >= 1, LSA_ERR_ARGUMENT);
  LSA_REQUIRE(!bucket_pages || (bucket_page_rows >= 1 && bucket_max_pages >= 1), LSA_ERR_ARGUMENT);
  LSA_REQUIRE(owner_world <= 1 || (owner_granule >= 1 && owner_rank >= 0 && owner_rank < owner_world),
              LSA_ERR_ARGUMENT);
  LSA_REQUIRE((int64_t)top_k + window + sink < INT32_MAX, LSA_ERR_ARGUMENT);
  if (R == 0) return LSA_OK;
  lsa::ExpandParams p = {};
  p.picked = picked;
  p.positions = positions;
  p.members = members;
  p.row_top_p = row_top_p;
  p.row_top_k = row_top_k;
  p.page_table = page_table;
  p.selected = selected;
  p.lengths = lengths;
  p.status = status;
  p.R = R;
  p.m = m;
  p.owner_first = owner_first;
  p.owner_end = owner_end;
  p.granule = owner_granule;
  p.world = owner_world;
  p.rank = owner_rank;
  p.flags = flags;
  p.row_request = row_request;
  p.page_table_stride = page_table_stride;
  p.bucket_pages = bucket_pages;
  p.bucket_pages_stride = bucket_pages_stride;
  p.bucket_max_pages = bucket_max_pages;
  p.bucket_page_rows = bucket_page_rows;
  p.top_p = top_p;
  p.cap = bucket_cap;
  p.top_k = top_k;
  p.sink = sink;
  p.window = window;
  p.page_size = page_size;
  p.width = top_k + window + sink;
  const bool keeps_all = owner_world <= 1 && owner_first <= 0 && owner_end == INT64_MAX;
  p.keeps_all = keeps_all;
  p.cap_inverse = ((1u << 21) + (uint32_t)bucket_cap - 1) / (uint32_t)bucket_cap;
  if (keeps_all && lsa::expands_spread(R, top_p, bucket_cap, window)) return lsa::launch_spread(p, (cudaStream_t)stream);  // (a decode step's long lists)
  // Many rows of long runs: a CTA a row (8,192 rows of 128 picks of 640 ids: 1,391 -> 459 us against a warp a row; 777 rows:
  // 497 -> 70 us). Short rows do not pay for the CTA's scan.
  if (keeps_all && top_p <= lsa::kRunMaxPicks && bucket_cap > lsa::kFlatCap && (int64_t)top_p * bucket_cap >= 8192) {
    lsa::expand_run_kernel<<<(unsigned)R, lsa::kRunThreads, 0, (cudaStream_t)stream>>>(p);
    LSA_LAUNCH_CHECK();
    return LSA_OK;
  }
  const unsigned grid = (unsigned)((R + lsa::kExpandWarps - 1) / lsa::kExpandWarps);
  lsa::launch(R <= lsa::kChainedRows, lsa::expand_kernel, dim3(grid), dim3(lsa::kExpandWarps * 32), 0,
              (cudaStream_t)stream, p);
  LSA_LAUNCH_CHECK();
  return LSA_OK;
}

LSA_API int lsa_expand(const int32_t *picked, int64_t R, int top_p, const int64_t *positions,
                       const int32_t *members, int64_t m, int bucket_cap, const int32_t *row_top_p,
                       const int32_t *row_top_k, int top_k, int sink, int window, const int32_t *page_table,
                       int page_size, int64_t owner_first, int64_t owner_end, int owner_granule, int owner_world,
                       int owner_rank, int flags, int32_t *selected, int32_t *lengths, int32_t *status,
                       void *stream) {
  return lsa_expand_batched(picked, R, top_p, positions, members, m, bucket_cap, row_top_p, row_top_k, top_k, sink,
                            window, page_table, page_size, owner_first, owner_end, owner_granule, owner_world,
                            owner_rank, flags, nullptr, 0, nullptr, 0, 0, 0, selected, lengths, status, stream);
}
