// Whether the rows of a matrix are unit vectors: one pass over it, two words out. (As a norm, a difference, its magnitude, a
// maximum and two passes for what is not finite the check of 1M rows of 64 dims took 0.49 ms; HBM-bound, 256 MB, it takes 46 us.)
#include "common.cuh"

namespace lsa {

constexpr int kUnitThreads = 256;

// out[0] = 1 where every element is finite, else 0; out[1] the greatest | |row| - 1 | (rows whose norm is no number count for
// nothing). LANES lanes a row, four elements a load where VEC, else one.
template <typename T, int LANES, bool VEC>
__global__ void __launch_bounds__(kUnitThreads)
    unit_rows_kernel(const T *__restrict__ rows, int64_t n, int d, float *__restrict__ out) {
  constexpr int kRows = 32 / LANES;  // of a warp at a time
  const int lane = lane_id(), at = lane % LANES;
  const int64_t step = (int64_t)gridDim.x * (kUnitThreads / 32) * kRows;
  bool finite = true;
  float most = 0.0f;
  for (int64_t r0 = ((int64_t)blockIdx.x * (kUnitThreads / 32) + (threadIdx.x >> 5)) * kRows; r0 < n; r0 += step) {
    const int64_t r = r0 + lane / LANES;
    const T *row = rows + r * d;
    float sum = 0.0f;
    auto take = [&](float x) {
      finite = finite && isfinite(x);
      sum = fmaf(x, x, sum);
    };
    if (r < n) {
      if constexpr (VEC) {
        for (int k = 4 * at; k < d; k += 4 * LANES) {
          if constexpr (sizeof(T) == 4) {
            const float4 x = __ldg(reinterpret_cast<const float4 *>(row + k));
            take(x.x), take(x.y), take(x.z), take(x.w);
          } else {
            const uint2 x = __ldg(reinterpret_cast<const uint2 *>(row + k));
            take(__uint_as_float(x.x << 16)), take(__uint_as_float(x.x & 0xFFFF0000u));
            take(__uint_as_float(x.y << 16)), take(__uint_as_float(x.y & 0xFFFF0000u));
          }
        }
      } else {
        for (int k = at; k < d; k += LANES) take(load_as_float(row, k));
      }
    }
#pragma unroll
    for (int o = LANES / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    const float off = fabsf(sqrtf(sum) - 1.0f);
    if (r < n && off > most) most = off;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, o));
  const bool good = __all_sync(0xffffffffu, finite);
  if (lane == 0) {
    if (most > 0.0f) atomicMax(reinterpret_cast<int *>(out) + 1, __float_as_int(most));  // (not negative: ordered as integers)
    if (!good) out[0] = 0.0f;
  }
}

__global__ void unit_rows_start_kernel(float *out) { out[0] = 1.0f, out[1] = 0.0f; }

}  // namespace lsa

LSA_API int lsa_unit_rows(const void *rows, int dtype, int64_t n, int d, float *out, void *stream) {
  LSA_REQUIRE(rows && out, LSA_ERR_NULL);
  LSA_REQUIRE(n >= 0 && d >= 1 && (dtype == LSA_DTYPE_F32 || dtype == LSA_DTYPE_BF16), LSA_ERR_ARGUMENT);
  cudaStream_t s = (cudaStream_t)stream;
  lsa::unit_rows_start_kernel<<<1, 1, 0, s>>>(out);
  LSA_LAUNCH_CHECK();
  if (n == 0) return LSA_OK;
  const int64_t most = 8 * (int64_t)lsa::sm_count(), want = (n + 15) / 16;
  const unsigned grid = (unsigned)(want < most ? want : most);
  const size_t bytes = dtype == LSA_DTYPE_F32 ? 4 : 2;
  const bool vec = d % 4 == 0 && ((uintptr_t)rows % (4 * bytes)) == 0;
  auto run = [&](auto kernel, const auto *typed) { kernel<<<grid, lsa::kUnitThreads, 0, s>>>(typed, n, d, out); };
  if (dtype == LSA_DTYPE_F32) {
    const float *x = (const float *)rows;
    if (vec && d <= 64)
      run(lsa::unit_rows_kernel<float, 16, true>, x);
    else if (vec)
      run(lsa::unit_rows_kernel<float, 32, true>, x);
    else
      run(lsa::unit_rows_kernel<float, 32, false>, x);
  } else {
    const uint16_t *x = (const uint16_t *)rows;
    if (vec)
      run(lsa::unit_rows_kernel<uint16_t, 16, true>, x);
    else
      run(lsa::unit_rows_kernel<uint16_t, 32, false>, x);
  }
  LSA_LAUNCH_CHECK();
  return LSA_OK;
}
