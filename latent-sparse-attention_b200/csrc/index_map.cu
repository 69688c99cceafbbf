// Index space: grouped-query head sum, learned linear map and row normalisation in one pass over the heads.
//
// out[s] = normalize( sum_kv (sum_{g < group} x[s, kv*group + g, off : off + dh_used]) @ W[kv*dh_used : (kv+1)*dh_used] )
// with fp32 accumulation, in ascending input-dim order except for a few rows (up to 32, or 128 under a bf16 map), whose threads
// share a row's dims. This is the exact-arithmetic form; rows are read once and the head sum never reaches memory.
#include <cooperative_groups.h>

#include "common.cuh"
#include "mma.cuh"

namespace lsa {

namespace cg = cooperative_groups;

constexpr int kMapThreads = 256;
constexpr int kMapRows = 64;    // rows a CTA maps, two a thread (half of them, one a thread, where 64 leave SMs without a second CTA)
constexpr int kMapSlice = 64;   // input dims staged at a time
constexpr int kMapMaxCols = 16; // output dims a thread holds: a CTA writes a slice of up to 128 output dims
constexpr int kMapColSlice = 8 * kMapMaxCols;

// COLS: output dims a thread holds. What bounds it is the chain of a slice: staging, 64 multiply-adds on one sum, and back. A
// slice whose columns are all there is unrolled, so that the shared-memory loads run ahead of the chain (7,613 rows of 256 dims
// to 64 121.8 -> 42.1 us, 200 of them 120 -> 34; 100,000 of 1,024 dims to 128 2.77 -> 1.48 ms).
template <typename TX, typename TW, int ROWS, int COLS>
__global__ void __launch_bounds__(kMapThreads)
    index_map_kernel(const TX *__restrict__ x, int64_t rows, int heads, int group, int dh_off, int dh_used,
                     int64_t x_row_stride, int64_t x_head_stride, const TW *__restrict__ W, int d_idx, int normalize,
                     float *__restrict__ out_f32, uint16_t *__restrict__ out_bf16) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float *xs = reinterpret_cast<float *>(smem_raw);       // [ROWS][kMapSlice + 1]
  float *ws = xs + ROWS * (kMapSlice + 1);           // [kMapSlice][d_idx]
  const int tid = threadIdx.x;
  const int row_a = tid >> 3, row_b = row_a + 32, cg = tid & 7;
  const int64_t row0 = (int64_t)blockIdx.x * ROWS;
  constexpr bool kTwo = ROWS == 64;  // whether a thread has a second row
  const int d_in = heads / group * dh_used;
  // blockIdx.y picks the slice of output dims; a map wider than one slice is normalised by a second kernel
  const int col0 = blockIdx.y * kMapColSlice, width = min(kMapColSlice, d_idx - col0);
  const int cols = (width + 7) / 8;
  float acc_a[COLS], acc_b[COLS];
#pragma unroll
  for (int i = 0; i < COLS; ++i) acc_a[i] = acc_b[i] = 0.0f;

  for (int k0 = 0; k0 < d_in; k0 += kMapSlice) {
    const int kn = min(kMapSlice, d_in - k0);
    // (loads of several elements in flight: one after another, each a round trip of the heads, they were most of the kernel)
#pragma unroll 4
    for (int e = tid; e < ROWS * kMapSlice; e += kMapThreads) {
      const int rr = e / kMapSlice, kk = e - rr * kMapSlice;
      float sum = 0.0f;
      const int64_t r = row0 + rr;
      if (r < rows && kk < kn) {
        const int k = k0 + kk, kv = k / dh_used, c = k - kv * dh_used;
        const TX *src = x + r * x_row_stride + (int64_t)kv * group * x_head_stride + dh_off + c;
#pragma unroll 8
        for (int g = 0; g < group; ++g) sum = __fadd_rn(sum, load_as_float<TX>(src, (int64_t)g * x_head_stride));
      }
      xs[rr * (kMapSlice + 1) + kk] = sum;
    }
#pragma unroll 8
    for (int e = tid; e < kMapSlice * width; e += kMapThreads) {
      const int kk = e / width, j = col0 + e - kk * width;
      float w = 0.0f;
      if (kk < kn) w = W ? load_as_float<TW>(W, (int64_t)(k0 + kk) * d_idx + j) : (k0 + kk == j ? 1.0f : 0.0f);
      ws[e] = w;
    }
    __syncthreads();
    if (width == 8 * COLS && kn == kMapSlice) {
#pragma unroll 8
      for (int kk = 0; kk < kMapSlice; ++kk) {
        const float xa = xs[row_a * (kMapSlice + 1) + kk], xb = kTwo ? xs[row_b * (kMapSlice + 1) + kk] : 0.0f;
        const float *wrow = ws + kk * 8 * COLS + cg;
#pragma unroll
        for (int i = 0; i < COLS; ++i) {
          acc_a[i] = fmaf(xa, wrow[8 * i], acc_a[i]);
          if (kTwo) acc_b[i] = fmaf(xb, wrow[8 * i], acc_b[i]);
        }
      }
      __syncthreads();
      continue;
    }
    for (int kk = 0; kk < kn; ++kk) {
      const float xa = xs[row_a * (kMapSlice + 1) + kk], xb = kTwo ? xs[row_b * (kMapSlice + 1) + kk] : 0.0f;
      const float *wrow = ws + kk * width + cg;
#pragma unroll
      for (int i = 0; i < COLS; ++i) {
        if (i < cols) {
          const float w = (cg + 8 * i) < width ? wrow[8 * i] : 0.0f;
          acc_a[i] = fmaf(xa, w, acc_a[i]);
          if (kTwo) acc_b[i] = fmaf(xb, w, acc_b[i]);
        }
      }
    }
    __syncthreads();
  }

  float ss_a = 0.0f, ss_b = 0.0f;
#pragma unroll
  for (int i = 0; i < COLS; ++i) {
    ss_a = fmaf(acc_a[i], acc_a[i], ss_a);
    ss_b = fmaf(acc_b[i], acc_b[i], ss_b);
  }
#pragma unroll
  for (int o = 1; o < 8; o <<= 1) {
    ss_a += __shfl_xor_sync(0xffffffffu, ss_a, o);
    ss_b += __shfl_xor_sync(0xffffffffu, ss_b, o);
  }
  const float den_a = normalize ? fmaxf(sqrtf(ss_a), 1e-12f) : 1.0f;
  const float den_b = normalize ? fmaxf(sqrtf(ss_b), 1e-12f) : 1.0f;
#pragma unroll
  for (int i = 0; i < COLS; ++i) {
    const int j = col0 + cg + 8 * i;
    if (i >= cols || cg + 8 * i >= width) continue;
    if (row0 + row_a < rows) {
      const float v = acc_a[i] / den_a;
      if (out_f32) out_f32[(row0 + row_a) * d_idx + j] = v;
      if (out_bf16) out_bf16[(row0 + row_a) * d_idx + j] = float_to_bf16_bits(v);
    }
    if (kTwo && row0 + row_b < rows) {
      const float v = acc_b[i] / den_b;
      if (out_f32) out_f32[(row0 + row_b) * d_idx + j] = v;
      if (out_bf16) out_bf16[(row0 + row_b) * d_idx + j] = float_to_bf16_bits(v);
    }
  }
}

// A few rows under a map that is not bf16 of 32, 64 or 128 columns: one CTA a row, its threads splitting the input dims, so the map of a single query
// is not one thread block walking the whole contraction alone.
constexpr int kRowThreads = 256;

template <typename TX, typename TW, int COLS>
__global__ void __launch_bounds__(kRowThreads)
    index_map_rows_kernel(const TX *__restrict__ x, int heads, int group, int dh_off, int dh_used, int64_t x_row_stride,
                          int64_t x_head_stride, const TW *__restrict__ W, int d_idx, int normalize,
                          float *__restrict__ out_f32, uint16_t *__restrict__ out_bf16) {
  __shared__ float partial[kRowThreads / 32][COLS];
  __shared__ float total[COLS];
  __shared__ float norm_s;
  const int64_t row = blockIdx.x;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int d_in = heads / group * dh_used;
  float acc[COLS];
#pragma unroll
  for (int j = 0; j < COLS; ++j) acc[j] = 0.0f;
  for (int k = tid; k < d_in; k += kRowThreads) {
    const int kv = k / dh_used, c = k - kv * dh_used;
    const TX *src = x + row * x_row_stride + (int64_t)kv * group * x_head_stride + dh_off + c;
    float xs = 0.0f;
#pragma unroll 8
    for (int g = 0; g < group; ++g) xs = __fadd_rn(xs, load_as_float<TX>(src, (int64_t)g * x_head_stride));
#pragma unroll
    for (int j = 0; j < COLS; ++j)
      if (j < d_idx) acc[j] = fmaf(xs, W ? load_as_float<TW>(W, (int64_t)k * d_idx + j) : (k == j ? 1.0f : 0.0f), acc[j]);
  }
  // The warp's sums of all columns at once: at every step a lane hands half of its columns to its partner and adds the
  // other half up (the pairs, and so the bits, of a shuffled sum a column, in 62 shuffles for 64 columns and not 320).
  int col = 0;
#pragma unroll
  for (int o = 16, n = COLS; o > 0; o >>= 1, n >>= 1) {
    const bool upper = lane & o;
#pragma unroll
    for (int i = 0; i < n / 2; ++i) {
      const float give = upper ? acc[i] : acc[i + n / 2], keep = upper ? acc[i + n / 2] : acc[i];
      acc[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
    }
    if (upper) col += n / 2;
  }
#pragma unroll
  for (int i = 0; i < COLS / 32; ++i) partial[warp][col + i] = acc[i];
  __syncthreads();
  if (tid < COLS) {
    float v = 0.0f;
    for (int w = 0; w < kRowThreads / 32; ++w) v += partial[w][tid];
    total[tid] = tid < d_idx ? v : 0.0f;
  }
  __syncthreads();
  if (tid == 0) {
    float ss = 0.0f;
    for (int j = 0; j < d_idx; ++j) ss = fmaf(total[j], total[j], ss);
    norm_s = normalize ? fmaxf(sqrtf(ss), 1e-12f) : 1.0f;
  }
  __syncthreads();
  if (tid < d_idx) {
    const float v = total[tid] / norm_s;
    if (out_f32) out_f32[row * d_idx + tid] = v;
    if (out_bf16) out_bf16[row * d_idx + tid] = float_to_bf16_bits(v);
  }
}

// The same for a bf16 map of 32, 64 or 128 columns: a CTA of 1,024 threads a row, so that the row's heads are one
// round of loads and the map's 128 KB another, both on their way at once. COLS / 8 neighbouring lanes take a row of the map,
// sixteen bytes each (a warp's load is 512 bytes in a run, where a lane that took a whole row of it touched a line a load),
// against the head sums in shared memory. What bounds it is the latency of those two rounds and of three barriers: a row of
// 5,120 dims to 64 takes 5.0 us (8.9 with a lane a row of the map), and 128 rows 5.4 (26.8 as one tile of the tensor-core map,
// whose CTA walks the 5,120 dims alone).
constexpr int kFewThreads = 1024, kFewHeld = 8, kFewRows = 128, kFewDims = 32 * 1024;

template <typename TX, int COLS>
__global__ void __launch_bounds__(kFewThreads, 1)
    index_map_few_kernel(const TX *__restrict__ x, int group, int dh_off, int dh_used, int64_t x_row_stride,
                         int64_t x_head_stride, const uint16_t *__restrict__ W, int d_in, int normalize,
                         float *__restrict__ out_f32, uint16_t *__restrict__ out_bf16) {
  constexpr int LANES = COLS / 8, DIMS = 32 / LANES, WARPS = kFewThreads / 32;  // lanes a map row, map rows a warp's load
  extern __shared__ __align__(16) float sums_s[];  // [d_in] the row's heads added up
  __shared__ float partial_s[WARPS][COLS];
  const int64_t row = blockIdx.x;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int first = warp * DIMS + lane / LANES, cols = lane % LANES * 8;
  const bool runs = ((uintptr_t)W % 16) == 0;
  auto run = [&](int k) {
    const uint16_t *w = W + (int64_t)k * COLS + cols;
    if (runs) return *reinterpret_cast<const uint4 *>(w);
    uint32_t w2[4];  // (a map that starts anywhere)
#pragma unroll
    for (int j = 0; j < 4; ++j) w2[j] = (uint32_t)w[2 * j] | (uint32_t)w[2 * j + 1] << 16;
    return make_uint4(w2[0], w2[1], w2[2], w2[3]);
  };
  uint4 held[kFewHeld];
#pragma unroll
  for (int i = 0; i < kFewHeld; ++i) {
    const int k = first + i * WARPS * DIMS;
    held[i] = k < d_in ? run(k) : make_uint4(0u, 0u, 0u, 0u);
  }
  for (int k = tid; k < d_in; k += kFewThreads) {
    const int kv = k / dh_used, c = k - kv * dh_used;
    const TX *src = x + row * x_row_stride + (int64_t)kv * group * x_head_stride + dh_off + c;
    float sum = 0.0f;
#pragma unroll 8
    for (int g = 0; g < group; ++g) sum = __fadd_rn(sum, load_as_float<TX>(src, (int64_t)g * x_head_stride));
    sums_s[k] = sum;
  }
  __syncthreads();
  float acc[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) acc[j] = 0.0f;
  auto fold = [&](const uint4 w, float by) {
    const uint32_t w2[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      acc[2 * j] = fmaf(by, __uint_as_float(w2[j] << 16), acc[2 * j]);
      acc[2 * j + 1] = fmaf(by, __uint_as_float(w2[j] & 0xFFFF0000u), acc[2 * j + 1]);
    }
  };
#pragma unroll
  for (int i = 0; i < kFewHeld; ++i) {
    const int k = first + i * WARPS * DIMS;
    if (k < d_in) fold(held[i], sums_s[k]);
  }
#pragma unroll 4
  for (int k = first + kFewHeld * WARPS * DIMS; k < d_in; k += WARPS * DIMS) fold(run(k), sums_s[k]);
#pragma unroll
  for (int o = LANES; o < 32; o <<= 1)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], o);
  if (lane < LANES) {
#pragma unroll
    for (int j = 0; j < 8; ++j) partial_s[warp][cols + j] = acc[j];
  }
  __syncthreads();
  if (warp > 0) return;
  float v[COLS / 32], ss = 0.0f;
#pragma unroll
  for (int i = 0; i < COLS / 32; ++i) {
    float part[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
    for (int w = 0; w < WARPS; ++w) part[w & 3] += partial_s[w][lane + 32 * i];
    v[i] = (part[0] + part[1]) + (part[2] + part[3]);
    ss = fmaf(v[i], v[i], ss);
  }
  const float den = normalize ? fmaxf(sqrtf(warp_sum(ss)), 1e-12f) : 1.0f;
#pragma unroll
  for (int i = 0; i < COLS / 32; ++i) {
    const int64_t at = row * COLS + lane + 32 * i;
    const float unit = v[i] / den;
    if (out_f32) out_f32[at] = unit;
    if (out_bf16) out_bf16[at] = float_to_bf16_bits(unit);
  }
}

// Unit rows in place, a warp a row: the second pass of a map wider than one slice.
__global__ void __launch_bounds__(256)
    rownorm_kernel(float *__restrict__ rows, int64_t n, int d, uint16_t *__restrict__ out_bf16) {
  const int64_t row = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (row >= n) return;
  float *r = rows + row * d;
  float ss = 0.0f;
  for (int j = lane; j < d; j += 32) ss = fmaf(r[j], r[j], ss);
  ss = warp_sum(ss);
  const float den = fmaxf(sqrtf(ss), 1e-12f);
  for (int j = lane; j < d; j += 32) {
    const float v = r[j] / den;
    r[j] = v;
    if (out_bf16) out_bf16[row * d + j] = float_to_bf16_bits(v);
  }
}

// The head sum alone (no map, no normalisation): out[r, kv*dh_used + c] = sum_g x[r, kv*group + g, off + c], added in
// head order - what the identity map computes, without walking a contraction.
template <typename TX>
__global__ void __launch_bounds__(256)
    head_sum_kernel(const TX *__restrict__ x, int64_t rows, int d_in, int group, int dh_off, int dh_used,
                    int64_t x_row_stride, int64_t x_head_stride, float *__restrict__ out_f32,
                    uint16_t *__restrict__ out_bf16) {
  const int64_t e = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (e >= rows * d_in) return;
  const int64_t r = e / d_in;
  const int k = (int)(e - r * d_in), kv = k / dh_used, c = k - kv * dh_used;
  const TX *src = x + r * x_row_stride + (int64_t)kv * group * x_head_stride + dh_off + c;
  float sum = 0.0f;
  for (int g = 0; g < group; ++g) sum = __fadd_rn(sum, load_as_float<TX>(src, (int64_t)g * x_head_stride));
  if (out_f32) out_f32[e] = sum;
  if (out_bf16) out_bf16[e] = float_to_bf16_bits(sum);
}

template <typename TX, typename TW>
static int launch_index_map(const void *x, int64_t rows, int heads, int group, int dh_off, int dh_used,
                            int64_t x_row_stride, int64_t x_head_stride, const void *W, int d_idx, int normalize,
                            float *out_f32, uint16_t *out_bf16, cudaStream_t s) {
  if (!W && !normalize) {
    const int64_t total = rows * d_idx;
    head_sum_kernel<TX><<<(unsigned)((total + 255) / 256), 256, 0, s>>>(
        (const TX *)x, rows, d_idx, group, dh_off, dh_used, x_row_stride, x_head_stride, out_f32, out_bf16);
    LSA_LAUNCH_CHECK();
    return LSA_OK;
  }
  const int d_in = heads / group * dh_used;
  if (rows <= kFewRows && sizeof(TW) == 2 && W && (d_idx == 32 || d_idx == 64 || d_idx == 128) && d_in <= kFewDims) {
    auto few = d_idx == 32 ? index_map_few_kernel<TX, 32> : d_idx == 64 ? index_map_few_kernel<TX, 64> : index_map_few_kernel<TX, 128>;
    if (!allow_shared(few, kFewDims * sizeof(float))) return LSA_ERR_LAUNCH;
    few<<<(unsigned)rows, kFewThreads, (size_t)d_in * sizeof(float), s>>>(
        (const TX *)x, group, dh_off, dh_used, x_row_stride, x_head_stride, (const uint16_t *)W, d_in, normalize, out_f32,
        out_bf16);
    LSA_LAUNCH_CHECK();
    return LSA_OK;
  }
  if (rows <= 32 && d_idx <= 128) {
    if (d_idx <= 64)
      index_map_rows_kernel<TX, TW, 64><<<(unsigned)rows, kRowThreads, 0, s>>>(
          (const TX *)x, heads, group, dh_off, dh_used, x_row_stride, x_head_stride, (const TW *)W, d_idx, normalize,
          out_f32, out_bf16);
    else
      index_map_rows_kernel<TX, TW, 128><<<(unsigned)rows, kRowThreads, 0, s>>>(
          (const TX *)x, heads, group, dh_off, dh_used, x_row_stride, x_head_stride, (const TW *)W, d_idx, normalize,
          out_f32, out_bf16);
    LSA_LAUNCH_CHECK();
    return LSA_OK;
  }
  const int slices = (d_idx + kMapColSlice - 1) / kMapColSlice;
  const bool half = (rows + kMapRows - 1) / kMapRows * slices < 2 * sm_count();
  const int cta_rows = half ? kMapRows / 2 : kMapRows;
  const size_t smem =
      sizeof(float) * ((size_t)cta_rows * (kMapSlice + 1) + (size_t)kMapSlice * min(d_idx, kMapColSlice));
  auto of = [&](auto whole, auto halves) { return half ? halves : whole; };
  auto kernel = d_idx <= 32   ? of(index_map_kernel<TX, TW, kMapRows, 4>, index_map_kernel<TX, TW, kMapRows / 2, 4>)
                : d_idx <= 64 ? of(index_map_kernel<TX, TW, kMapRows, 8>, index_map_kernel<TX, TW, kMapRows / 2, 8>)
                              : of(index_map_kernel<TX, TW, kMapRows, kMapMaxCols>, index_map_kernel<TX, TW, kMapRows / 2, kMapMaxCols>);
  if (!allow_shared(kernel, sizeof(float) * (kMapRows * (kMapSlice + 1) + (size_t)kMapSlice * kMapColSlice)))
    return LSA_ERR_LAUNCH;
  const dim3 grid((unsigned)((rows + cta_rows - 1) / cta_rows), (unsigned)slices);
  // One slice: the CTA holds whole rows and normalises them itself. More: fp32 rows first, then unit rows in place.
  kernel<<<grid, kMapThreads, smem, s>>>(
      (const TX *)x, rows, heads, group, dh_off, dh_used, x_row_stride, x_head_stride, (const TW *)W, d_idx,
      slices == 1 ? normalize : 0, out_f32, slices == 1 || !normalize ? out_bf16 : nullptr);
  LSA_LAUNCH_CHECK();
  if (slices > 1 && normalize) {
    rownorm_kernel<<<(unsigned)((rows + 7) / 8), 256, 0, s>>>(out_f32, rows, d_idx, out_bf16);
    LSA_LAUNCH_CHECK();
  }
  return LSA_OK;
}

// A linear layer over a FEW rows (a decode step's queries): out[r, n] = act(sum_k xs[r, k] Wt[n, k]), xs = the row's
// heads summed (fp32, rounded once to bf16) or the row itself. A warp owns an output column and walks its weights once
// for all rows; eight columns a CTA, so even a single row's map spreads over N / 8 CTAs instead of one.
constexpr int kLinMaxRows = 8, kLinUnitCols = 64;  // (columns of a map whose grid is one cluster)
constexpr size_t kLinStaged = 96 * 1024;  // a row's heads are staged whole where they take no more than this
// 16-byte runs of a column's weights a lane takes before anything else: 8 (2,048 weights a column), or 20 (5,120) for
// the widest maps - the kernel is built for both, so that a narrow map does not carry the registers of a wide one.

// STAGED: a row's heads come into shared memory in one round of asynchronous copies and are added from there, in head order
// (sixteen warps a CTA then: every CTA sums the heads for itself, 73 KB of them for 64 heads of 576 dims into 2,048 columns:
// 7.8 us with two dependent rounds of a thread's own loads, 4.4 this way; 8 rows 30.6 and 21.7).
template <int kLinHeld, bool STAGED>
__global__ void __launch_bounds__(STAGED ? 512 : 256)
    rows_linear_kernel(const uint16_t *__restrict__ x, int rows, int heads, int64_t x_row_stride, int64_t x_head_stride,
                       int K, const uint16_t *__restrict__ Wt, int N, int gelu, int unit, float *__restrict__ out_f32,
                       uint16_t *__restrict__ out_bf16) {
  constexpr int kLinThreads = STAGED ? 512 : 256;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ float whole_s[kLinMaxRows][kLinUnitCols];  // the whole rows, where the grid is a cluster that makes them unit rows
  uint16_t *xs = reinterpret_cast<uint16_t *>(smem_raw);  // [rows][K] bf16
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (unit) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");  // (waited for before the first write there)
  dependents_may_launch();
  // The weights of this warp's column do not depend on the kernel before: up to 5,120 of them are taken first, while
  // that kernel may still be running (where the launch is chained).
  const int n = blockIdx.x * (kLinThreads / 32) + warp;
  uint4 held[kLinHeld];
#pragma unroll
  for (int i = 0; i < kLinHeld; ++i) {
    const int k = lane * 8 + i * 256;
    held[i] = n < N && k < K ? *reinterpret_cast<const uint4 *>(Wt + (int64_t)n * K + k) : make_uint4(0, 0, 0, 0);
  }
  wait_for_earlier_grids();
  // the head sum: a thread a pair of dims, 32 heads' loads in flight at a time, added in head order
  const bool pairs = (K % 2 == 0) && (x_row_stride % 2 == 0) && (x_head_stride % 2 == 0) && ((uintptr_t)x % 4 == 0);
  if constexpr (STAGED) {
    const int per_head = K / 8;
    const uint32_t staged = smem_u32(xs + rows * K);
    const uint32_t *staged_pairs = reinterpret_cast<const uint32_t *>(xs + rows * K);
    for (int r = 0; r < rows; ++r) {
      if (r > 0) __syncthreads();  // (the last row's heads have been added)
      for (int e = tid; e < heads * per_head; e += kLinThreads) {
        const int h = e / per_head;
        cp_async_16(staged + e * 16, x + (int64_t)r * x_row_stride + (int64_t)h * x_head_stride + (e - h * per_head) * 8, 16);
      }
      cp_async_commit();
      cp_async_wait<0>();
      __syncthreads();
      for (int k = tid; k < K / 2; k += kLinThreads) {
        float lo = 0.0f, hi = 0.0f;
#pragma unroll 16
        for (int h = 0; h < heads; ++h) {
          const uint32_t v = staged_pairs[h * (K / 2) + k];
          lo = __fadd_rn(lo, __uint_as_float(v << 16));
          hi = __fadd_rn(hi, __uint_as_float(v & 0xFFFF0000u));
        }
        reinterpret_cast<uint32_t *>(xs + r * K)[k] = pack_bf16x2(lo, hi);
      }
    }
  } else if (heads == 1 && x_row_stride % 8 == 0 && ((uintptr_t)x % 16) == 0) {
    // nothing to sum: the rows are copied 16 bytes a thread, four loads in flight (K is a multiple of 8)
    const int per_row = K / 8, total = rows * per_row;
    for (int e0 = tid; e0 < total; e0 += 4 * kLinThreads) {
      uint4 v[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int e = e0 + j * kLinThreads, r = e / per_row, c = e - r * per_row;
        if (e < total) v[j] = *reinterpret_cast<const uint4 *>(x + (int64_t)r * x_row_stride + c * 8);
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int e = e0 + j * kLinThreads;
        if (e < total) reinterpret_cast<uint4 *>(xs)[e] = v[j];
      }
    }
  } else if (pairs) {
    for (int e = tid; e < rows * (K / 2); e += kLinThreads) {
      const int r = e / (K / 2), k = 2 * (e - r * (K / 2));
      const uint16_t *src = x + (int64_t)r * x_row_stride + k;
      float lo = 0.0f, hi = 0.0f;
      for (int h0 = 0; h0 < heads; h0 += 32) {
        uint32_t v[32];
#pragma unroll
        for (int j = 0; j < 32; ++j)
          v[j] = h0 + j < heads ? *reinterpret_cast<const uint32_t *>(src + (int64_t)(h0 + j) * x_head_stride) : 0u;
#pragma unroll
        for (int j = 0; j < 32; ++j)
          if (h0 + j < heads) {
            lo = __fadd_rn(lo, __uint_as_float(v[j] << 16));
            hi = __fadd_rn(hi, __uint_as_float(v[j] & 0xFFFF0000u));
          }
      }
      if (heads > 1) {
        xs[r * K + k] = float_to_bf16_bits(lo), xs[r * K + k + 1] = float_to_bf16_bits(hi);
      } else {
        xs[r * K + k] = src[0], xs[r * K + k + 1] = src[1];
      }
    }
  } else {
    for (int e = tid; e < rows * K; e += kLinThreads) {
      const int r = e / K, k = e - r * K;
      const uint16_t *src = x + (int64_t)r * x_row_stride + k;
      float sum = 0.0f;
      for (int h = 0; h < heads; ++h) sum = __fadd_rn(sum, bf16_bits_to_float(src[(int64_t)h * x_head_stride]));
      xs[e] = heads > 1 ? float_to_bf16_bits(sum) : src[0];
    }
  }
  __syncthreads();
  if (n >= N && !unit) return;
  float acc[kLinMaxRows];
#pragma unroll
  for (int r = 0; r < kLinMaxRows; ++r) acc[r] = 0.0f;
  const uint16_t *w = Wt + (int64_t)n * K;
  // (K is a multiple of 8 and the rows are 16-byte aligned; a lane walks its weights in ascending order either way)
  auto fold = [&](const uint4 wv, int k) {
    const uint32_t wp[4] = {wv.x, wv.y, wv.z, wv.w};
#pragma unroll
    for (int r = 0; r < kLinMaxRows; ++r) {
      if (r >= rows) break;
      const uint4 xv = *reinterpret_cast<const uint4 *>(xs + r * K + k);
      const uint32_t xp[4] = {xv.x, xv.y, xv.z, xv.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        acc[r] = fmaf(__uint_as_float(xp[i] << 16), __uint_as_float(wp[i] << 16), acc[r]);
        acc[r] = fmaf(__uint_as_float(xp[i] & 0xFFFF0000u), __uint_as_float(wp[i] & 0xFFFF0000u), acc[r]);
      }
    }
  };
#pragma unroll
  for (int i = 0; i < kLinHeld; ++i) {
    const int k = lane * 8 + i * 256;
    if (k < K) fold(held[i], k);
  }
#pragma unroll 4
  for (int k = lane * 8 + kLinHeld * 256; n < N && k < K; k += 32 * 8) fold(*reinterpret_cast<const uint4 *>(w + k), k);
#pragma unroll
  for (int r = 0; r < kLinMaxRows; ++r) {
    if (r >= rows) break;
    float v = warp_sum(acc[r]);
    if (gelu) v = 0.5f * v * (1.0f + erff(v * 0.70710678118654752440f));
    if (unit) {
      acc[r] = v;
    } else if (lane == 0) {
      if (out_f32) out_f32[(int64_t)r * N + n] = v;
      if (out_bf16) out_bf16[(int64_t)r * N + n] = float_to_bf16_bits(v);
    }
  }
  if (unit) {
    // A map of few columns is one cluster: every CTA gets the whole rows and divides its own columns by their length, the sums
    // in rows_unit_kernel's order (a launch of its own was 1.9 us and the gap before it).
    cg::cluster_group cluster = cg::this_cluster();
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (n < N && lane < (int)gridDim.x) {
#pragma unroll
      for (int r = 0; r < kLinMaxRows; ++r)
        if (r < rows) *cluster.map_shared_rank(&whole_s[r][n], lane) = acc[r];
    }
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    const int first = blockIdx.x * (kLinThreads / 32);
    for (int r = warp; r < rows; r += kLinThreads / 32) {
      float ss = 0.0f;
      for (int j = lane; j < N; j += 32) ss = fmaf(whole_s[r][j], whole_s[r][j], ss);
      ss = warp_sum(ss);
      const float den = fmaxf(sqrtf(ss), 1e-12f);
      const int j = first + lane;
      if (lane < kLinThreads / 32 && j < N) {
        const float v = whole_s[r][j] / den;
        if (out_f32) out_f32[(int64_t)r * N + j] = v;
        if (out_bf16) out_bf16[(int64_t)r * N + j] = float_to_bf16_bits(v);
      }
    }
  }
}

// rows /= their length (fp32 in place, a warp a row), with an optional bf16 copy
__global__ void rows_unit_kernel(float *__restrict__ rows, int n_rows, int d, uint16_t *__restrict__ out_bf16) {
  dependents_may_launch();
  wait_for_earlier_grids();
  const int r = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (r >= n_rows) return;
  float ss = 0.0f;
  for (int j = lane; j < d; j += 32) ss = fmaf(rows[(int64_t)r * d + j], rows[(int64_t)r * d + j], ss);
  ss = warp_sum(ss);
  const float den = fmaxf(sqrtf(ss), 1e-12f);
  for (int j = lane; j < d; j += 32) {
    const float v = rows[(int64_t)r * d + j] / den;
    rows[(int64_t)r * d + j] = v;
    if (out_bf16) out_bf16[(int64_t)r * d + j] = float_to_bf16_bits(v);
  }
}

}  // namespace lsa

LSA_API int lsa_rows_linear(const uint16_t *x, int rows, int heads, int64_t x_row_stride, int64_t x_head_stride,
                            int d_in, const uint16_t *Wt, int d_out, int flags, float *out_f32, uint16_t *out_bf16,
                            void *stream) {
  LSA_REQUIRE(x && Wt && (out_f32 || out_bf16), LSA_ERR_NULL);
  LSA_REQUIRE(rows >= 0 && rows <= lsa::kLinMaxRows && heads >= 1 && d_in >= 8 && d_in % 8 == 0 && d_out >= 1,
              LSA_ERR_ARGUMENT);
  LSA_REQUIRE(((uintptr_t)Wt % 16) == 0, LSA_ERR_ARGUMENT);
  LSA_REQUIRE(!(flags & LSA_ROWS_NORMALIZE) || out_f32, LSA_ERR_ARGUMENT);
  size_t smem = (size_t)rows * d_in * 2;
  constexpr size_t most = 160 * 1024;
  LSA_REQUIRE(smem <= most, LSA_ERR_UNSUPPORTED);
  if (rows == 0) return LSA_OK;
  const size_t heads_bytes = (size_t)heads * d_in * 2;
  const bool staged = heads > 1 && d_in <= 2048 && heads_bytes <= lsa::kLinStaged && smem + heads_bytes <= most &&
                      x_row_stride % 8 == 0 && x_head_stride % 8 == 0 && ((uintptr_t)x % 16) == 0;
  if (staged) smem += heads_bytes;
  auto kernel = staged ? lsa::rows_linear_kernel<8, true>
                       : d_in <= 2048 ? lsa::rows_linear_kernel<8, false> : lsa::rows_linear_kernel<20, false>;
  if (!lsa::allow_shared(kernel, most)) return LSA_ERR_LAUNCH;
  const unsigned threads = staged ? 512 : 256, grid = (unsigned)((d_out + threads / 32 - 1) / (threads / 32));
  const bool unit = flags & LSA_ROWS_NORMALIZE;
  // (a grid of up to eight CTAs is a cluster that makes its rows unit rows itself. It is never chained to the kernel before: 64
  // heads through 2,048 columns to 64, a graph under LSA_CHAINED_LAUNCH=1, both layers: 7.4 us so, 8.9 as a dependent; 8.3 unchained)
  const bool clustered = unit && !staged && d_out <= lsa::kLinUnitCols;
  const int gelu = flags & LSA_ROWS_GELU ? 1 : 0;
  uint16_t *const half = unit && !clustered ? nullptr : out_bf16;
  if (clustered) {
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(grid), config.blockDim = dim3(threads), config.dynamicSmemBytes = smem, config.stream = (cudaStream_t)stream;
    cudaLaunchAttribute attribute[1];
    attribute[0].id = cudaLaunchAttributeClusterDimension;
    attribute[0].val.clusterDim.x = grid, attribute[0].val.clusterDim.y = attribute[0].val.clusterDim.z = 1;
    config.attrs = attribute, config.numAttrs = 1;
    (void)cudaLaunchKernelEx(&config, kernel, x, rows, heads, x_row_stride, x_head_stride, d_in, Wt, d_out, gelu, 1, out_f32, half);
    LSA_LAUNCH_CHECK();
    return LSA_OK;
  }
  lsa::launch(true, kernel, dim3(grid), dim3(threads), smem, (cudaStream_t)stream, x, rows,
              heads, x_row_stride, x_head_stride, d_in, Wt, d_out, gelu, 0, out_f32, half);
  LSA_LAUNCH_CHECK();
  if (unit) {
    lsa::launch(true, lsa::rows_unit_kernel, dim3((unsigned)((rows + 3) / 4)), dim3(128), 0, (cudaStream_t)stream,
                out_f32, rows, d_out, out_bf16);
    LSA_LAUNCH_CHECK();
  }
  return LSA_OK;
}

LSA_API int lsa_index_map(const void *x, int x_dtype, int64_t rows, int heads, int group, int dh_off, int dh_used,
                          int64_t x_row_stride, int64_t x_head_stride, const void *W, int w_dtype, int d_idx,
                          int normalize, float *out_f32, uint16_t *out_bf16, void *stream) {
  LSA_REQUIRE(x && (out_f32 || out_bf16), LSA_ERR_NULL);
  LSA_REQUIRE(rows >= 0 && heads >= 1 && group >= 1 && heads % group == 0 && dh_off >= 0 && dh_used >= 1 &&
                  d_idx >= 1,
              LSA_ERR_ARGUMENT);
  LSA_REQUIRE(x_dtype == LSA_DTYPE_F32 || x_dtype == LSA_DTYPE_BF16, LSA_ERR_ARGUMENT);
  LSA_REQUIRE(w_dtype == LSA_DTYPE_F32 || w_dtype == LSA_DTYPE_BF16, LSA_ERR_ARGUMENT);
  LSA_REQUIRE(W || d_idx == heads / group * dh_used, LSA_ERR_ARGUMENT);
  // a map wider than one slice of output dims is normalised in place in its fp32 output
  LSA_REQUIRE(d_idx <= lsa::kMapColSlice || !normalize || out_f32, LSA_ERR_UNSUPPORTED);
  if (rows == 0) return LSA_OK;
  cudaStream_t s = (cudaStream_t)stream;
  if (x_dtype == LSA_DTYPE_BF16 && w_dtype == LSA_DTYPE_BF16)
    return lsa::launch_index_map<uint16_t, uint16_t>(x, rows, heads, group, dh_off, dh_used, x_row_stride,
                                                     x_head_stride, W, d_idx, normalize, out_f32, out_bf16, s);
  if (x_dtype == LSA_DTYPE_BF16)
    return lsa::launch_index_map<uint16_t, float>(x, rows, heads, group, dh_off, dh_used, x_row_stride,
                                                  x_head_stride, W, d_idx, normalize, out_f32, out_bf16, s);
  if (w_dtype == LSA_DTYPE_BF16)
    return lsa::launch_index_map<float, uint16_t>(x, rows, heads, group, dh_off, dh_used, x_row_stride,
                                                  x_head_stride, W, d_idx, normalize, out_f32, out_bf16, s);
  return lsa::launch_index_map<float, float>(x, rows, heads, group, dh_off, dh_used, x_row_stride, x_head_stride, W,
                                             d_idx, normalize, out_f32, out_bf16, s);
}
