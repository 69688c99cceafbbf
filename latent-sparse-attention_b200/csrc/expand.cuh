// What a decode step's scan and its expansion share: the expansion is a launch of its own or the tail of the scan, the last merge of
// a scan's lists a launch of its own or the head of the expansion.
#pragma once

#include "common.cuh"

namespace lsa {

// How many of list[0..size) (descending, size a power of two) come before `key`: those greater, and equal ones too if `ties`.
__device__ __forceinline__ int keys_before(const int64_t *list, int size, int64_t key, bool ties) {
  int at = 0;
  for (int step = size >> 1; step; step >>= 1) {
    const int64_t other = list[at + step - 1];
    at += other > key || (ties && other == key) ? step : 0;
  }
  const int64_t other = list[at];
  return at + (other > key || (ties && other == key) ? 1 : 0);
}

// The run of N buckets' members that lie from the sinks on and before the window: where it starts in the bucket's row and how many
// there are. Members ascend, so a warp looks at 32 places spread over a row and then at the places between two of them: two rounds
// of loads, those of the N buckets in flight together. `at`: where a bucket's row starts in the member table, -1 for none.
template <int N>
__device__ __forceinline__ void member_runs(const int32_t *members, int cap, const int64_t (&at)[N], int64_t window_start, int sink,
                                            int (&first)[N], int (&count)[N]) {
  const int lane = lane_id(), step = (cap + 31) / 32;
  auto before_window = [&](int32_t id) { return id >= 0 && id < window_start; };
  int32_t sample[N], head[N];
#pragma unroll
  for (int j = 0; j < N; ++j) {
    // the last place of each 32nd of the row, and the row's first 32 places
    const int place = min(cap, (lane + 1) * step) - 1;
    sample[j] = at[j] >= 0 && lane * step < cap ? members[at[j] + place] : LSA_PAD;
    head[j] = at[j] >= 0 && lane < cap ? members[at[j] + lane] : LSA_PAD;
  }
  int whole[N];  // 32nds that lie before the window
  int32_t inner[N];
#pragma unroll
  for (int j = 0; j < N; ++j) {
    whole[j] = __popc(__ballot_sync(0xffffffffu, before_window(sample[j])));
    const int place = whole[j] * step + lane;
    inner[j] = at[j] >= 0 && lane < step && place < cap ? members[at[j] + place] : LSA_PAD;
  }
#pragma unroll
  for (int j = 0; j < N; ++j) {
    int end = min(cap, whole[j] * step) + __popc(__ballot_sync(0xffffffffu, before_window(inner[j])));
    for (int l0 = 32; l0 < step; l0 += 32) {  // (rows of more than 1,024 places)
      const int place = whole[j] * step + l0 + lane;
      const int32_t id = at[j] >= 0 && l0 + lane < step && place < cap ? members[at[j] + place] : LSA_PAD;
      end += __popc(__ballot_sync(0xffffffffu, before_window(id)));
    }
    int begin = __popc(__ballot_sync(0xffffffffu, head[j] >= 0 && head[j] < sink));
    if (begin == 32)  // (more sinks in the bucket than that: one after another)
      while (begin < end && members[at[j] + begin] < sink) ++begin;
    first[j] = min(begin, end), count[j] = end - first[j];
  }
}

// Exclusive sums of n counts, and all of them at starts[n]; by one warp.
__device__ __forceinline__ void run_starts(const int *counts, int n, int *starts) {
  const int lane = lane_id();
  int carry = 0;
  for (int base = 0; base < n; base += 32) {
    const int v = base + lane < n ? counts[base + lane] : 0;
    int incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += up;
    }
    if (base + lane < n) starts[base + lane] = carry + incl - v;
    carry += __shfl_sync(0xffffffffu, incl, 31);
  }
  if (lane == 0) starts[n] = carry;
}

// The ids of a list's places first, first + step, .. under `listed`, out of the picks' runs: the pick whose run a place lies in by
// bisection of the runs' starts, four loads in flight. `put(place, id)` takes each.
template <typename Put>
__device__ __forceinline__ void list_members(const int32_t *members, const int64_t *from, const int *starts, int picks, int listed,
                                             int first, int step, Put put) {
  constexpr int kAhead = 4;
  for (int e0 = first; e0 < listed; e0 += kAhead * step) {
    int32_t ids[kAhead];
#pragma unroll
    for (int j = 0; j < kAhead; ++j) {
      const int e = e0 + j * step;
      ids[j] = LSA_PAD;
      if (e < listed) {
        int lo = 0, hi = picks;  // the last pick whose run starts at or before e
        while (hi - lo > 1) {
          const int mid = (lo + hi) >> 1;
          if (starts[mid] <= e) lo = mid; else hi = mid;
        }
        ids[j] = members[from[lo] + (e - starts[lo])];
      }
    }
#pragma unroll
    for (int j = 0; j < kAhead; ++j) {
      const int e = e0 + j * step;
      if (e < listed) put(e, ids[j]);
    }
  }
}

// Where a scan of a few rows leaves its rows' read lists instead of their picks (lsa_expand's lists, without a page table, ranges or
// padding).
struct RowLists {
  const int32_t *members;  // [m, cap]
  int32_t *lists;          // [R, width]
  int32_t *lengths;        // [R]
  int64_t width;
  int cap, top_k, sink, window;
};

// Whether rows of such picks are expanded by several CTAs each (expand_spread_kernel), and that expansion over the picks of `parts`
// lists a row, sorted keys [parts][R][top_p]: the best top_p of them all.
bool expands_spread(int64_t R, int top_p, int cap, int window);
int expand_sorted(const int64_t *keys, int parts, int64_t R, int top_p, const int64_t *positions, int64_t m, const RowLists &to,
                  cudaStream_t stream);

}  // namespace lsa
