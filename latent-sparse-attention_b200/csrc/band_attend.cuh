// What the dense reads share: the tensor-memory kernel's parameters and its launch (band_attend_tc.cu).
#pragma once

#include "common.cuh"

namespace lsa {

struct BandTcParams {
  float *out, *lse;          // fp32 output and log-sum-exp, either may be NULL
  uint16_t *out_bf16;        // or NULL
  const uint4 *mask;         // [key tiles][R] a bit a key of the tile: the keys that a row reads; NULL: window and sinks
  int32_t *not_finite;       // set where a row's output is not finite, or NULL
  int32_t *status;
  int R, n_keys, first_position;  // (positions fit 31 bits)
  int Hq, group, window, sink;
  float scale_log2;
};

struct BandTcCall {
  const uint16_t *q, *k, *v;
  int64_t q_row_stride, kv_row_stride;
  int Hkv;
  BandTcParams p;
};

// The caller has checked dh == 128, heads packed densely and the alignments a tensor map needs.
int launch_band_attend_tc(const BandTcCall &call, cudaStream_t stream);

}  // namespace lsa
