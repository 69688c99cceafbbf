// The exact flat search of a prefill chunk in two passes: every row's scores into a scratch matrix, a few thousand rows at a time
// so that it stays in the L2, and each row's best out of it by counting. Key for key lsa_flat_select's other forms.
//
// Scores: a CTA of 64 rows by 128 buckets, a warp eight rows, a lane four buckets. Multiply-adds are fma.rn.f32x2 - two
// neighbouring buckets' sums, each the scalar chain in ascending dim order -, with a row's values twice and the values of two
// buckets side by side in shared memory, so that no operand has to be put together.
//
// Best: a CTA a row. Scores fall into bins by value, greatest first (one multiply, monotone; the bins split the row's own range);
// a scan of the bins' counts finds the bin that holds the last one kept; the keys of the bins up to it are laid out bin by bin, and
// a key's place is its bin's first place plus how many keys of its bin beat it. Nothing is sorted. Where a bin holds more than its
// share (a score far from all others leaves them one bin), the bins split the range of that bin's scores, with what lies above and
// below it in the first and the last, or where those are one score the range of their ids; what two such rounds do not spread is
// sorted.
//
// What bounds it is a CTA's chain of passes and barriers a row, six CTAs an SM side by side (eight up to 2,048 buckets; a row's keys
// have room for the last resort's sort, a power of two of them); the scores are a fifth of it. 8,192
// rows of 64 dims over 3,072 buckets, one B200: top 1,024 990 us as a warp a row that cut and sorted its buffer in one CTA of eight
// warps an SM, 222 so; top 64 291 and 172; equal scores 958 and 232.
#include "common.cuh"
#include "mma.cuh"

namespace lsa {

constexpr int kScoreRows = 64, kScoreCols = 128, kScoreThreads = 256;
constexpr int kBinThreads = 256, kBins = 4 * kBinThreads;
constexpr int kBinMost = 160;          // keys of a bin that are placed by counting, at most
constexpr int kBinnedBuckets = 4096;   // buckets, at most: the keys of a row lie in shared memory, 32 KB
constexpr size_t kBinnedScratch = 48u << 20;

// Scores as ordered integers [rows, ld]; buckets that no row of a CTA sees are left out.
template <int D>
__global__ void __launch_bounds__(kScoreThreads, 2)
    exact_scores_kernel(const float *__restrict__ queries, const float *__restrict__ centroids, const int32_t *__restrict__ visible,
                        int64_t rows, int m, int ld, int32_t *__restrict__ scores) {
  constexpr int kRows = kScoreRows / (kScoreThreads / 32), kPairs = kScoreCols / 64, kLd = 2 * D + 4;
  extern __shared__ __align__(16) float score_s[];
  float *a = score_s, *b = score_s + kScoreRows * 2 * D;  // [64][D] twice each; [64 pairs][kLd]
  __shared__ int widest_s;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int64_t row0 = (int64_t)blockIdx.y * kScoreRows;
  const int col0 = (int)blockIdx.x * kScoreCols;
  if (tid == 0) widest_s = 0;
  __syncthreads();
  if (tid < kScoreRows && row0 + tid < rows) atomicMax(&widest_s, visible[row0 + tid]);
  __syncthreads();
  if (col0 >= widest_s) return;
  for (int e = tid; e < kScoreRows * (D / 4); e += kScoreThreads) {
    const int r = e / (D / 4), k = e - r * (D / 4);
    if (row0 + r >= rows) continue;
    const float4 x = *reinterpret_cast<const float4 *>(queries + (row0 + r) * D + 4 * k);
    *reinterpret_cast<float4 *>(a + r * 2 * D + 8 * k) = make_float4(x.x, x.x, x.y, x.y);
    *reinterpret_cast<float4 *>(a + r * 2 * D + 8 * k + 4) = make_float4(x.z, x.z, x.w, x.w);
  }
  for (int e = tid; e < kScoreCols / 2 * (D / 4); e += kScoreThreads) {
    const int r = e / (D / 4), k = e - r * (D / 4), c = col0 + 2 * r;
    if (c >= m) continue;
    const float4 x = __ldg(reinterpret_cast<const float4 *>(centroids + (int64_t)c * D) + k);
    const float4 y = __ldg(reinterpret_cast<const float4 *>(centroids + (int64_t)min(c + 1, m - 1) * D) + k);
    *reinterpret_cast<float4 *>(b + r * kLd + 8 * k) = make_float4(x.x, y.x, x.y, y.y);
    *reinterpret_cast<float4 *>(b + r * kLd + 8 * k + 4) = make_float4(x.z, y.z, x.w, y.w);
  }
  __syncthreads();
  uint64_t acc[kRows][kPairs];
#pragma unroll
  for (int i = 0; i < kRows; ++i)
#pragma unroll
    for (int j = 0; j < kPairs; ++j) acc[i][j] = 0ull;
#pragma unroll 4
  for (int k = 0; k < D; k += 2) {
    ulonglong2 y[kPairs];
#pragma unroll
    for (int j = 0; j < kPairs; ++j) y[j] = *reinterpret_cast<const ulonglong2 *>(b + (lane + 32 * j) * kLd + 2 * k);
#pragma unroll
    for (int i = 0; i < kRows; ++i) {
      const ulonglong2 x = *reinterpret_cast<const ulonglong2 *>(a + (warp * kRows + i) * 2 * D + 2 * k);
#pragma unroll
      for (int j = 0; j < kPairs; ++j) {
        acc[i][j] = fma_pair(x.x, y[j].x, acc[i][j]);
        acc[i][j] = fma_pair(x.y, y[j].y, acc[i][j]);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < kRows; ++i) {
    const int64_t row = row0 + warp * kRows + i;
    if (row >= rows) break;
#pragma unroll
    for (int j = 0; j < kPairs; ++j) {
      float lo, hi;
      split_pair(acc[i][j], lo, hi);
      const int c = col0 + 2 * (lane + 32 * j);
      if (c < ld) *reinterpret_cast<int2 *>(scores + row * ld + c) = make_int2(ordered_bits(lo), ordered_bits(hi));  // (ld is even)
    }
  }
}

struct BinParams {
  const int32_t *scores;             // [rows, ld]
  const int32_t *visible, *row_keep;  // [rows]; row_keep or NULL
  int64_t *keys_out;
  int32_t *ids_out;
  int ld, m, keep, id_base;
};

constexpr int32_t kLeastScore = (int32_t)(0xFF7FFFFFu ^ 0x7FFFFFFFu);  // the least and (-1 less it) the greatest finite score, ordered
__device__ __forceinline__ float score_of(int32_t ordered) {
  return __int_as_float(ordered < 0 ? (ordered ^ 0x7FFFFFFF) : ordered);
}

__global__ void __launch_bounds__(kBinThreads) bin_select_kernel(BinParams p) {
  extern __shared__ __align__(16) int64_t area[];  // the keys of the bins that hold the best ones
  __shared__ __align__(16) int bins_s[kBins];      // counts (read four at a time), then where the next key of a bin goes
  __shared__ int low_s, high_s, most_s, last_s, count_s, sums_s[kBinThreads / 32];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int64_t row = blockIdx.x;
  const int n = min(max(p.visible[row], 0), p.m);
  const int keep = min(p.row_keep ? max(0, min(p.row_keep[row], p.keep)) : p.keep, n);
  int64_t *keys_out = p.keys_out ? p.keys_out + row * p.keep : nullptr;
  int32_t *ids_out = p.ids_out ? p.ids_out + row * p.keep : nullptr;
  auto write = [&](int at, int64_t key) {
    if (keys_out) keys_out[at] = key;
    if (ids_out) ids_out[at] = key_id(key);
  };
  for (int i = keep + tid; i < p.keep; i += kBinThreads) {
    if (keys_out) keys_out[i] = kEmptyKey;
    if (ids_out) ids_out[i] = LSA_PAD;
  }
  if (keep == 0) return;
  const int32_t *scores = p.scores + row * p.ld;
  if (tid == 0) low_s = INT32_MAX, high_s = INT32_MIN;
  __syncthreads();
  // the scores of `within`, the least and the greatest (numbers: what is none lies above or below all bins)
  auto find_range = [&](auto within) {
    int32_t low = INT32_MAX, high = INT32_MIN;
    for (int i = tid; i < n; i += kBinThreads) {
      const int32_t v = __ldg(scores + i);
      if (v >= kLeastScore && v <= -1 - kLeastScore && within(v, i)) low = min(low, v), high = max(high, v);
    }
    low = __reduce_min_sync(0xffffffffu, low), high = __reduce_max_sync(0xffffffffu, high);
    if (lane == 0) atomicMin(&low_s, low), atomicMax(&high_s, high);
    __syncthreads();
  };
  find_range([](int32_t, int) { return true; });
  int32_t low, high;
  float top, scale;
  bool by_id;
  // Which bin a score belongs to: the inner ones split low .. high, or where those are one number the ids.
  auto bin_of = [&](int32_t v, int i) {
    if (v > high) return 0;
    if (v < low) return kBins - 1;
    const int inner = by_id ? (int)((float)i * scale) : (int)((top - score_of(v)) * scale);
    return 1 + min(inner, kBins - 3);
  };
  for (int round = 0;; ++round) {
    low = low_s, high = high_s;
    top = score_of(high);
    const float range = top - score_of(low);
    by_id = low >= high;  // (of the ordered integers, as the keys have them: -0 and +0 are two scores, in one bin)
    scale = (float)(kBins - 2) / (by_id ? (float)n : range);
    if (!isfinite(scale)) scale = 0.0f;
#pragma unroll
    for (int i = 0; i < kBins / kBinThreads; ++i) bins_s[tid + i * kBinThreads] = 0;
    if (tid == 0) most_s = 0;
    __syncthreads();
    for (int i = tid; i < n; i += kBinThreads) atomicAdd(&bins_s[bin_of(__ldg(scores + i), i)], 1);
    __syncthreads();
    // where each bin starts (four neighbouring bins a thread), the bin that holds the last key kept, the fullest up to it
    {
      const int4 own = *reinterpret_cast<const int4 *>(bins_s + 4 * tid);
      const int sum = own.x + own.y + own.z + own.w;
      int incl = sum;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += up;
      }
      if (lane == 31) sums_s[warp] = incl;
      __syncthreads();
      int at = incl - sum;
#pragma unroll
      for (int w = 0; w < kBinThreads / 32; ++w) at += w < warp ? sums_s[w] : 0;
      const int counts[4] = {own.x, own.y, own.z, own.w};
      int most = 0;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        bins_s[4 * tid + j] = at;
        if (at < keep) {
          most = max(most, counts[j] * kBins + 4 * tid + j);
          if (at + counts[j] >= keep) last_s = 4 * tid + j, count_s = at + counts[j];
        }
        at += counts[j];
      }
      most = __reduce_max_sync(0xffffffffu, most);
      if (lane == 0) atomicMax(&most_s, most);
    }
    __syncthreads();
    if (most_s / kBins <= kBinMost || round == 2) break;
    const int fullest = most_s % kBins;
    if (fullest == 0 || fullest == kBins - 1) break;  // (more than a few scores that are no numbers)
    if (tid == 0) low_s = INT32_MAX, high_s = INT32_MIN;
    __syncthreads();
    find_range([&](int32_t v, int i) { return bin_of(v, i) == fullest; });
  }
  const int last = last_s, count = count_s;
  for (int i = tid; i < n; i += kBinThreads) {
    const int32_t v = __ldg(scores + i);
    const int bin = bin_of(v, i);
    if (bin > last) continue;
    area[atomicAdd(&bins_s[bin], 1)] = (int64_t)((uint64_t)(uint32_t)v << 32) | (uint32_t)(0x7FFFFFFF - (i + p.id_base));
  }
  __syncthreads();  // (a bin's entry is where it ends now)
  if (most_s / kBins <= kBinMost) {
    for (int i = tid; i < count; i += kBinThreads) {
      const int64_t key = area[i];
      const int bin = bin_of((int32_t)(key >> 32), key_id(key) - p.id_base), first = bin ? bins_s[bin - 1] : 0, end = bins_s[bin];
      int rank = first;
      for (int j = first; j < end; ++j) rank += area[j] > key;
      if (rank < keep) write(rank, key);
    }
    return;
  }
  int size = 1;
  while (size < count) size <<= 1;
  for (int i = count + tid; i < size; i += kBinThreads) area[i] = kEmptyKey;
  for (int span = 2; span <= size; span <<= 1)
    for (int stride = span >> 1; stride > 0; stride >>= 1) {
      __syncthreads();
      for (int t = tid; t < size / 2; t += kBinThreads) {
        const int i = ((t & ~(stride - 1)) << 1) | (t & (stride - 1)), j = i | stride;
        const int64_t x = area[i], y = area[j];
        if ((x < y) == ((i & span) == 0)) area[i] = y, area[j] = x;
      }
    }
  __syncthreads();
  for (int i = tid; i < keep; i += kBinThreads) write(i, area[i]);
}

// Rows of the scratch, and a row's pitch in it.
static int binned_pitch(int64_t m) { return (int)((m + 3) & ~(int64_t)3); }
static int64_t binned_rows(int64_t R, int64_t m) {
  const int64_t fit = (int64_t)(kBinnedScratch / ((size_t)binned_pitch(m) * 4)) / kScoreRows * kScoreRows;
  return R < fit ? R : fit;
}

template <int D>
static int run_binned(const float *queries, int64_t R, const float *centroids, int64_t m, const int32_t *visible,
                      const int32_t *row_top_p, int top_p, int32_t id_base, int64_t *keys_out, int32_t *picked_out, int32_t *scratch,
                      cudaStream_t s) {
  constexpr size_t smem = (size_t)(kScoreRows * 2 * D + kScoreCols / 2 * (2 * D + 4)) * 4;
  size_t size = 1;
  while (size < (size_t)m) size <<= 1;
  if (!allow_shared(exact_scores_kernel<D>, smem) || !allow_shared(bin_select_kernel, (size_t)kBinnedBuckets * 8)) return LSA_ERR_LAUNCH;
  const int ld = binned_pitch(m);
  const int64_t most = binned_rows(R, m);
  for (int64_t r0 = 0; r0 < R; r0 += most) {
    const int64_t rows = R - r0 < most ? R - r0 : most;
    const dim3 grid((unsigned)((m + kScoreCols - 1) / kScoreCols), (unsigned)((rows + kScoreRows - 1) / kScoreRows));
    exact_scores_kernel<D><<<grid, kScoreThreads, smem, s>>>(queries + r0 * D, centroids, visible + r0, rows, (int)m, ld, scratch);
    LSA_LAUNCH_CHECK();
    const BinParams p = {scratch, visible + r0, row_top_p ? row_top_p + r0 : nullptr, keys_out ? keys_out + r0 * top_p : nullptr,
                         picked_out ? picked_out + r0 * top_p : nullptr, ld, (int)m, top_p, id_base};
    bin_select_kernel<<<(unsigned)rows, kBinThreads, size * 8, s>>>(p);
    LSA_LAUNCH_CHECK();
  }
  return LSA_OK;
}

}  // namespace lsa

LSA_API size_t lsa_flat_select_binned_workspace_bytes(int64_t R, int d, int64_t m) {
  if (R <= 0 || m <= 0 || m > lsa::kBinnedBuckets || (d != 32 && d != 64)) return 0;
  return (size_t)lsa::binned_rows(R, m) * lsa::binned_pitch(m) * 4;
}

LSA_API int lsa_flat_select_binned(const float *queries, int64_t R, int d, const float *centroids, int64_t m,
                                   const int32_t *visible, const int32_t *row_top_p, int top_p, int32_t bucket_id_base,
                                   int64_t *keys_out, int32_t *picked_out, void *workspace, size_t workspace_bytes, void *stream) {
  LSA_REQUIRE(queries && centroids && visible && (keys_out || picked_out) && workspace, LSA_ERR_NULL);
  LSA_REQUIRE(R >= 0 && m >= 0 && top_p >= 1, LSA_ERR_ARGUMENT);
  LSA_REQUIRE((d == 32 || d == 64) && m >= 1 && m <= lsa::kBinnedBuckets && ((uintptr_t)queries % 16) == 0 &&
                  ((uintptr_t)centroids % 16) == 0 && ((uintptr_t)workspace % 16) == 0,
              LSA_ERR_UNSUPPORTED);
  if (R == 0) return LSA_OK;
  LSA_REQUIRE(workspace_bytes >= lsa_flat_select_binned_workspace_bytes(R, d, m), LSA_ERR_WORKSPACE);
  const auto run = d == 64 ? lsa::run_binned<64> : lsa::run_binned<32>;
  return run(queries, R, centroids, m, visible, row_top_p, top_p, bucket_id_base, keys_out, picked_out, (int32_t *)workspace,
             (cudaStream_t)stream);
}
