// The local part of a prefill's read - each query's sliding window and the sinks - as dense banded attention.
//
// Consecutive query rows read almost the same recent keys, so unlike the selected keys (one gather a row) the window
// is a shared band: a CTA takes 16 consecutive query rows of one KV head, one warp a query head of the group, and
// streams the band's K/V tiles (64 keys) through shared memory once for all of them. Scores and the weighted sum run
// on mma.m16n8k16 with the queries as M; softmax is online in fp32. The result is a PARTIAL read: normalised output
// and log-sum-exp per (row, head), which lsa_sparse_attend takes as its starting state and extends with the
// gathered keys.
#include "band_attend.cuh"
#include "common.cuh"
#include "mma.cuh"

namespace lsa {

constexpr int kBandRows = 16;  // query rows a CTA
constexpr int kBandKeys = 64;  // keys a tile

struct BandParams {
  const uint16_t *q, *k, *v;
  float *out, *lse;
  int64_t R, n_keys, first_position, q_row_stride, q_head_stride, kv_row_stride, kv_head_stride;
  int Hq, Hkv, group, window, sink;
  float scale_log2;
};

// grid (ceil(R / 16), Hkv, ceil(group / 8)); blockDim = min(group, 8) * 32. Row i of the call sits at position first_position + i and KV
// row p holds position p.
// TWO_TERM: the probabilities enter the second product as bf16 and what bf16 left of them.
template <int DH, bool TWO_TERM>
__global__ void band_attend_kernel(BandParams p) {
  constexpr int ROW_BYTES = DH * 2, CHUNKS = ROW_BYTES / 16, KSTEPS = DH / 16;
  constexpr int TILE_BYTES = kBandKeys * ROW_BYTES;
  extern __shared__ __align__(128) unsigned char smem_raw[];  // 2 stages x (K tile, V tile)
  const uint32_t smem_base = smem_u32(smem_raw);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int64_t row0 = (int64_t)blockIdx.x * kBandRows;
  const int h = blockIdx.y;
  // At most eight heads of the group a CTA (blockIdx.z takes the rest); a warp past the group mirrors the last head
  // so that it still takes part in the loads and barriers, and writes nothing.
  const int in_group = blockIdx.z * 8 + warp;
  const bool real_head = in_group < p.group;
  const int head = h * p.group + (real_head ? in_group : p.group - 1);
  const int64_t pos0 = p.first_position + row0;              // position of the tile's first row
  const int64_t pos_last = min(pos0 + kBandRows - 1, p.first_position + p.R - 1);
  // The band of the tile: from the first row's window start to the last row, in whole tiles; tile -1 is the sinks.
  const int64_t band_first = max((int64_t)0, pos0 + 1 - p.window) / kBandKeys * kBandKeys;
  const int tiles = (int)((pos_last - band_first) / kBandKeys) + 1;
  const bool has_sinks = p.sink > 0 && band_first > 0;
  const int first_tile = has_sinks ? -1 : 0;
  const uint16_t *k_head = p.k + (int64_t)h * p.kv_head_stride, *v_head = p.v + (int64_t)h * p.kv_head_stride;

  auto load_tile = [&](int tile, int stage) {
    const int64_t key0 = tile < 0 ? 0 : band_first + (int64_t)tile * kBandKeys;
    const uint32_t dst0 = smem_base + stage * 2 * TILE_BYTES;
    for (int e = threadIdx.x; e < kBandKeys * CHUNKS; e += blockDim.x) {
      const int row = e / CHUNKS, chunk = e - row * CHUNKS;
      const int64_t key = key0 + row;
      const bool ok = key < p.n_keys && (tile >= 0 || row < p.sink);
      const int64_t off = ok ? key * p.kv_row_stride + chunk * 8 : 0;
      const uint32_t dst = dst0 + row * ROW_BYTES + ((chunk ^ (row & 7)) << 4);
      cp_async_16(dst, k_head + off, ok ? 16 : 0);
      cp_async_16(dst + TILE_BYTES, v_head + off, ok ? 16 : 0);
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };

  // Q as the A operand: thread (g, t) holds rows g and g + 8, dims t*2, t*2+1 (+8) of each 16-dim step.
  uint32_t qa[KSTEPS][4];
  {
    const int64_t ra = row0 + g, rb = row0 + g + 8;
    const uint16_t *qa_row = p.q + ra * p.q_row_stride + (int64_t)head * p.q_head_stride;
    const uint16_t *qb_row = p.q + rb * p.q_row_stride + (int64_t)head * p.q_head_stride;
#pragma unroll
    for (int ks = 0; ks < KSTEPS; ++ks) {
      const int c = ks * 16 + t * 2;
      qa[ks][0] = ra < p.R ? *reinterpret_cast<const uint32_t *>(qa_row + c) : 0u;
      qa[ks][1] = rb < p.R ? *reinterpret_cast<const uint32_t *>(qb_row + c) : 0u;
      qa[ks][2] = ra < p.R ? *reinterpret_cast<const uint32_t *>(qa_row + c + 8) : 0u;
      qa[ks][3] = rb < p.R ? *reinterpret_cast<const uint32_t *>(qb_row + c + 8) : 0u;
    }
  }
  float o[DH / 8][4];
#pragma unroll
  for (int n = 0; n < DH / 8; ++n) o[n][0] = o[n][1] = o[n][2] = o[n][3] = 0.0f;
  float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.0f, 0.0f};
  const int64_t pos_a = pos0 + g, pos_b = pos0 + g + 8;  // positions of this thread's two rows

  load_tile(first_tile, 0);
  for (int tile = first_tile; tile < tiles; ++tile) {
    const int stage = (tile - first_tile) & 1;
    if (tile + 1 < tiles) {
      load_tile(tile + 1, stage ^ 1);
      asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    }
    __syncthreads();
    const uint32_t k_src = smem_base + stage * 2 * TILE_BYTES, v_src = k_src + TILE_BYTES;
    const int64_t key0 = tile < 0 ? 0 : band_first + (int64_t)tile * kBandKeys;

    // S [16 rows x 64 keys] = Q K^T
    float s[kBandKeys / 8][4];
#pragma unroll
    for (int n = 0; n < kBandKeys / 8; ++n) s[n][0] = s[n][1] = s[n][2] = s[n][3] = 0.0f;
#pragma unroll
    for (int ks = 0; ks < KSTEPS; ++ks) {
#pragma unroll
      for (int np = 0; np < kBandKeys / 16; ++np) {
        const int row = np * 16 + (lane & 7) + (lane >> 4) * 8;
        const int chunk = ks * 2 + ((lane >> 3) & 1);
        uint32_t b0, b1, b2, b3;
        ldmatrix_x4(k_src + row * ROW_BYTES + ((chunk ^ (row & 7)) << 4), b0, b1, b2, b3);
        mma_bf16(s[2 * np], qa[ks][0], qa[ks][1], qa[ks][2], qa[ks][3], b0, b1);
        mma_bf16(s[2 * np + 1], qa[ks][0], qa[ks][1], qa[ks][2], qa[ks][3], b2, b3);
      }
    }
    // mask: a key counts for a row if it is inside the row's window (and causal), or one of its sinks. A tile that
    // lies inside every row's window (all but the band's two ends) needs none.
    float mx[2] = {-INFINITY, -INFINITY};
    const bool inside = tile >= 0 && key0 >= max((int64_t)0, pos_last + 1 - p.window) && key0 + kBandKeys - 1 <= pos0 &&
                        key0 + kBandKeys <= p.n_keys && pos0 + kBandRows <= p.first_position + p.R;
    if (inside) {
#pragma unroll
      for (int n = 0; n < kBandKeys / 8; ++n) {
#pragma unroll
        for (int j = 0; j < 4; ++j) mx[j >> 1] = fmaxf(mx[j >> 1], s[n][j]);
      }
    } else {
#pragma unroll
      for (int n = 0; n < kBandKeys / 8; ++n) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int64_t key = key0 + n * 8 + t * 2 + (j & 1);
          const int64_t pos = (j & 2) ? pos_b : pos_a;
          const int64_t start = max((int64_t)0, pos + 1 - p.window);
          const bool ok = pos < p.first_position + p.R && key < p.n_keys &&
                          ((tile >= 0 && key >= start && key <= pos) || key < min((int64_t)p.sink, start));
          s[n][j] = ok ? s[n][j] : -INFINITY;
          mx[j >> 1] = fmaxf(mx[j >> 1], s[n][j]);
        }
      }
    }
    float alpha[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 1));
      mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 2));
      // the products are raw: the scale is positive, so it is applied to the maximum and inside the exponent
      const float m_new = fmaxf(m_run[r], mx[r] * p.scale_log2);
      const float m_safe = m_new == -INFINITY ? 0.0f : m_new;
      alpha[r] = fast_exp2(m_run[r] - m_safe);
      m_run[r] = m_new;
      mx[r] = m_safe;
      l_run[r] *= alpha[r];
    }
#pragma unroll
    for (int n = 0; n < kBandKeys / 8; ++n) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        s[n][j] = fast_exp2(fmaf(s[n][j], p.scale_log2, -mx[j >> 1]));
        l_run[j >> 1] += s[n][j];
      }
    }
    // (once a row has met its largest keys the maximum stops moving and the rescale is a multiply by one)
    if (__any_sync(0xffffffffu, alpha[0] != 1.0f || alpha[1] != 1.0f)) {
#pragma unroll
      for (int n = 0; n < DH / 8; ++n) {
        o[n][0] *= alpha[0];
        o[n][1] *= alpha[0];
        o[n][2] *= alpha[1];
        o[n][3] *= alpha[1];
      }
    }
    // O [16 rows x DH] += P [16 x 64] V [64 x DH]
#pragma unroll
    for (int kk = 0; kk < kBandKeys / 16; ++kk) {
      const uint32_t a0 = pack_bf16x2(s[2 * kk][0], s[2 * kk][1]), a1 = pack_bf16x2(s[2 * kk][2], s[2 * kk][3]);
      const uint32_t a2 = pack_bf16x2(s[2 * kk + 1][0], s[2 * kk + 1][1]), a3 = pack_bf16x2(s[2 * kk + 1][2], s[2 * kk + 1][3]);
      auto left = [](const float *x, uint32_t w) {
        return pack_bf16x2(x[0] - __uint_as_float(w << 16), x[1] - __uint_as_float(w & 0xFFFF0000u));
      };
      uint32_t b[4] = {0u, 0u, 0u, 0u};
      if constexpr (TWO_TERM)
        b[0] = left(s[2 * kk], a0), b[1] = left(s[2 * kk] + 2, a1), b[2] = left(s[2 * kk + 1], a2),
        b[3] = left(s[2 * kk + 1] + 2, a3);
#pragma unroll
      for (int np = 0; np < DH / 16; ++np) {
        const int row = kk * 16 + (lane & 7) + ((lane >> 3) & 1) * 8;
        const int chunk = np * 2 + (lane >> 4);
        uint32_t b0, b1, b2, b3;
        ldmatrix_x4_trans(v_src + row * ROW_BYTES + ((chunk ^ (row & 7)) << 4), b0, b1, b2, b3);
        mma_bf16(o[2 * np], a0, a1, a2, a3, b0, b1);
        mma_bf16(o[2 * np + 1], a0, a1, a2, a3, b2, b3);
        if constexpr (TWO_TERM) {
          mma_bf16(o[2 * np], b[0], b[1], b[2], b[3], b0, b1);
          mma_bf16(o[2 * np + 1], b[0], b[1], b[2], b[3], b2, b3);
        }
      }
    }
    __syncthreads();
  }

  constexpr float kLn2 = 0.6931471805599453f;
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    float l = l_run[r];
    l += __shfl_xor_sync(0xffffffffu, l, 1);
    l += __shfl_xor_sync(0xffffffffu, l, 2);
    const int64_t row = row0 + g + r * 8;
    if (row >= p.R || !real_head) continue;
    const float inv = l > 0.0f ? 1.0f / l : 0.0f;
    float *dst = p.out + (row * p.Hq + head) * DH;
#pragma unroll
    for (int n = 0; n < DH / 8; ++n)
      *reinterpret_cast<float2 *>(dst + n * 8 + t * 2) = make_float2(o[n][2 * r] * inv, o[n][2 * r + 1] * inv);
    if (t == 0) p.lse[row * p.Hq + head] = l > 0.0f ? (m_run[r] + log2f(l)) * kLn2 : -INFINITY;
  }
}

struct RoundParams {
  const float *in;
  const uint16_t *q, *k, *v;
  uint16_t *out_bf16;
  float *out_f32;
  int64_t R, n_keys, first_position, q_row_stride, q_head_stride, kv_row_stride, kv_head_stride;
  int Hq, group;
  float scale_log2;
};

// A row's heads read again by a warp, HEADS of one KV head at a time: the keys up to the row's own, or those of them that `mask`
// (a bit a key, in tiles of 128 keys a row) names, 32 at once. A lane takes a key's scores, then DH / 32 dims of the sum. What
// bounds it is a warp's rounds of 32 keys: their loads, the products, the weights, the values, one after another. (4,096 causal
// rows of 16 heads with an infinity among their values 26.9 -> 4.7 ms, rows that list a quarter of the keys 11.1 -> 1.4, where a
// key at a time cost a warp 400 cycles of dependent loads, shuffles and exponentials; 0.12 each without the infinity.)
constexpr int kAgainHeads = 4, kAgainWarps = 4;

// A warp's shared memory. Several heads (a launch that may have every row to read) have the keys at hand staged there: lanes that
// read a key's row each from memory touch 32 lines a load (6.1 ms for the 4.7 above).
template <int DH, int HEADS>
struct __align__(16) AgainRoom {
  static constexpr bool kStaged = HEADS > 1;
  static constexpr int kPitch = DH + 8;  // (16 bytes on: eight lanes' reads of 16 bytes take all banks)
  float q[HEADS][DH];
  uint16_t k[kStaged ? 32 * kPitch : 8];
  float e[32][HEADS];  // the weights of the keys at hand
  int32_t ids[64];     // keys found and not yet read
};

template <int DH, int HEADS>
__device__ __noinline__ void read_again(const RoundParams &p, int64_t r, int head0, int heads, const uint32_t *mask,
                                        AgainRoom<DH, HEADS> &room, float (&out)[HEADS][DH / 32]) {
  constexpr int PER = DH / 32;
  const int lane = lane_id(), h = head0 / p.group;
  const uint16_t *q = p.q + r * p.q_row_stride + (int64_t)head0 * p.q_head_stride + lane * PER;
  const uint16_t *k = p.k + (int64_t)h * p.kv_head_stride, *v = p.v + (int64_t)h * p.kv_head_stride + lane * PER;
  const bool runs = ((uintptr_t)k % 16) == 0 && ((uintptr_t)v % (2 * PER)) == 0 && p.kv_row_stride % 8 == 0;
  auto word_at = [&](const uint16_t *at) {  // two neighbours
    return runs ? *reinterpret_cast<const uint32_t *>(at) : (uint32_t)at[0] | (uint32_t)at[1] << 16;
  };
  float m[HEADS], l[HEADS], x[HEADS][PER];
  __syncwarp();
#pragma unroll
  for (int g = 0; g < HEADS; ++g) {
    m[g] = -INFINITY, l[g] = 0.0f;
#pragma unroll
    for (int c = 0; c < PER; ++c) {
      x[g][c] = 0.0f;
      room.q[g][lane * PER + c] = g < heads ? bf16_bits_to_float(q[(int64_t)g * p.q_head_stride + c]) : 0.0f;
    }
  }
  const int64_t end = min(p.n_keys, p.first_position + r + 1);
  int64_t next = 0;         // the first key not looked at
  uint32_t word = 0;        // lane i: which of the keys next - 1024 + 32 i .. are read
  uint32_t pending = 0;     // the lanes whose words are still to be taken
  int held = 0;
  for (;;) {
    while (held < 32) {
      if (pending == 0) {
        if (next >= end) break;
        const int64_t key = next + 32 * lane;
        word = key >= end ? 0u : mask ? mask[((key >> 7) * p.R + r) * 4 + ((key >> 5) & 3)] : 0xffffffffu;
        if (key < end && key + 32 > end) word &= (1u << (int)(end - key)) - 1u;
        pending = __ballot_sync(0xffffffffu, word != 0);
        next += 32 * 32;
        continue;
      }
      const int from = __ffs(pending) - 1;
      pending &= pending - 1;
      const uint32_t taken = __shfl_sync(0xffffffffu, word, from);
      if (taken >> lane & 1) room.ids[held + __popc(taken & ((1u << lane) - 1u))] = (int32_t)(next - 32 * 32 + 32 * from + lane);
      held += __popc(taken);
    }
    if (held == 0) break;
    const int n = min(held, 32);
    __syncwarp();
    const uint16_t *row = k + (int64_t)room.ids[lane < n ? lane : 0] * p.kv_row_stride;
    if constexpr (AgainRoom<DH, HEADS>::kStaged) {
      constexpr int PIECES = DH / 8, PITCH = AgainRoom<DH, HEADS>::kPitch;
      for (int e = lane; e < n * PIECES; e += 32) {  // (the caller: rows are 16-byte aligned)
        const int at = e / PIECES, piece = e - at * PIECES;
        cp_async_16(smem_u32(&room.k[at * PITCH + piece * 8]), k + (int64_t)room.ids[at] * p.kv_row_stride + piece * 8, 16);
      }
      cp_async_commit();
      cp_async_wait<0>();
      __syncwarp();
      row = &room.k[(lane < n ? lane : 0) * PITCH];
    }
    uint64_t dot[HEADS];  // even and odd dims
#pragma unroll
    for (int g = 0; g < HEADS; ++g) dot[g] = 0;
#pragma unroll 4
    for (int c = 0; c < DH; c += 8) {
      const uint4 w = runs ? *reinterpret_cast<const uint4 *>(row + c)
                           : make_uint4(word_at(row + c), word_at(row + c + 2), word_at(row + c + 4), word_at(row + c + 6));
      const uint32_t w2[4] = {w.x, w.y, w.z, w.w};
      uint64_t k2[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) k2[i] = pair_of(__uint_as_float(w2[i] << 16), __uint_as_float(w2[i] & 0xffff0000u));
#pragma unroll
      for (int g = 0; g < HEADS; ++g)
#pragma unroll
        for (int i = 0; i < 4; i += 2) {
          const float4 a = *reinterpret_cast<const float4 *>(&room.q[g][c + 2 * i]);
          dot[g] = fma_pair(k2[i], pair_of(a.x, a.y), dot[g]);
          dot[g] = fma_pair(k2[i + 1], pair_of(a.z, a.w), dot[g]);
        }
    }
#pragma unroll
    for (int g = 0; g < HEADS; ++g) {
      float even, odd;
      split_pair(dot[g], even, odd);
      const float s = lane < n ? (even + odd) * p.scale_log2 : -INFINITY;
      float m_new = s;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) m_new = fmaxf(m_new, __shfl_xor_sync(0xffffffffu, m_new, o));
      m_new = fmaxf(m[g], m_new);
      const float m_safe = m_new == -INFINITY ? 0.0f : m_new;
      const float alpha = exp2f(m[g] - m_safe), e = lane < n ? exp2f(s - m_safe) : 0.0f;
      m[g] = m_new;
      l[g] = fmaf(l[g], alpha, warp_sum(e));
      room.e[lane][g] = e;
#pragma unroll
      for (int c = 0; c < PER; ++c) x[g][c] *= alpha;
    }
    __syncwarp();
    for (int j0 = 0; j0 < n; j0 += 8) {
      uint32_t w[8][PER / 2];
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int c = 0; c < PER; c += 2)
          w[i][c / 2] = j0 + i < n ? word_at(v + (int64_t)room.ids[j0 + i] * p.kv_row_stride + c) : 0u;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        if (j0 + i >= n) break;
#pragma unroll
        for (int g = 0; g < HEADS; ++g) {
          const float e = room.e[j0 + i][g];
#pragma unroll
          for (int c = 0; c < PER; c += 2) {
            x[g][c] = fmaf(e, __uint_as_float(w[i][c / 2] << 16), x[g][c]);
            x[g][c + 1] = fmaf(e, __uint_as_float(w[i][c / 2] & 0xffff0000u), x[g][c + 1]);
          }
        }
      }
    }
    const int32_t rest = room.ids[32 + lane];
    __syncwarp();
    held -= n;
    if (lane < held) room.ids[lane] = rest;
  }
#pragma unroll
  for (int g = 0; g < HEADS; ++g) {
    const float inv = l[g] > 0.0f ? 1.0f / l[g] : 0.0f;
#pragma unroll
    for (int c = 0; c < PER; ++c) out[g][c] = x[g][c] * inv;
  }
}

// The rows of a dense read whose output is not finite, read again: nothing but a look at a word where there are none. A key
// that a row does not read weighs zero in its tile, and zero times a value that is not finite is not a number.
__global__ void __launch_bounds__(kAgainWarps * 32, 4)
    dense_repair_kernel(RoundParams p, const uint32_t *mask, const int32_t *not_finite) {
  __shared__ AgainRoom<128, kAgainHeads> rooms[kAgainWarps];
  if (*not_finite == 0) return;
  const int lane = lane_id(), warp = threadIdx.x >> 5;
  const int blocks = (p.group + kAgainHeads - 1) / kAgainHeads, a_row = p.Hq / p.group * blocks;  // of heads
  for (int64_t item = (int64_t)blockIdx.x * kAgainWarps + warp; item < p.R * a_row; item += (int64_t)gridDim.x * kAgainWarps) {
    const int64_t r = item / a_row;
    const int of_row = (int)(item - r * a_row), in_group = of_row % blocks * kAgainHeads;
    const int head0 = of_row / blocks * p.group + in_group, heads = min(kAgainHeads, p.group - in_group);
    const int64_t at0 = (r * p.Hq + head0) * 128 + lane * 4;
    uint32_t odd = 0;  // the heads that are not finite
    for (int g = 0; g < heads; ++g) {
      const int64_t at = at0 + g * 128;
      bool finite = true;
#pragma unroll
      for (int c = 0; c < 4; ++c)
        finite = finite && isfinite(p.out_bf16 ? bf16_bits_to_float(p.out_bf16[at + c]) : p.out_f32[at + c]);
      if (!__all_sync(0xffffffffu, finite)) odd |= 1u << g;
    }
    if (odd == 0) continue;
    float x[kAgainHeads][4];
    read_again<128, kAgainHeads>(p, r, head0, heads, mask, rooms[warp], x);
#pragma unroll
    for (int g = 0; g < kAgainHeads; ++g) {
      if (!(odd >> g & 1)) continue;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        if (p.out_bf16) p.out_bf16[at0 + g * 128 + c] = float_to_bf16_bits(x[g][c]);
        if (p.out_f32) p.out_f32[at0 + g * 128 + c] = x[g][c];
      }
    }
  }
}

// A dense causal read on its way out (rounded to bf16, or as it is), a warp a (row, head). In a tile of 128 rows a key after a row weighs zero, and zero
// times a value that is not finite is not a number: a row of the tile that holds one is read again here, over the keys up to
// its own alone (what a list would name). Memory bounds the rows that are finite, all of them as a rule (six
// bytes a dim, what the copy to bf16 in its place moved).
template <int DH>
__global__ void __launch_bounds__(256) band_round_kernel(RoundParams p) {
  constexpr int PER = DH / 32;  // dims a lane holds
  const int lane = lane_id();
  const int64_t item = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (item >= p.R * p.Hq) return;
  float x[PER];
  bool finite = true;
#pragma unroll
  for (int c = 0; c < PER; ++c) x[c] = p.in[item * DH + lane * PER + c], finite = finite && isfinite(x[c]);
  __shared__ AgainRoom<DH, 1> rooms[8];
  if (!__all_sync(0xffffffffu, finite)) {
    float again[1][PER];
    read_again<DH, 1>(p, item / p.Hq, (int)(item % p.Hq), 1, nullptr, rooms[threadIdx.x >> 5], again);
#pragma unroll
    for (int c = 0; c < PER; ++c) x[c] = again[0][c];
  }
  const int64_t at = item * DH + lane * PER;
  if (p.out_f32) {
#pragma unroll
    for (int c = 0; c < PER; ++c) p.out_f32[at + c] = x[c];
  }
  if (p.out_bf16 && ((uintptr_t)p.out_bf16 & 3) == 0) {
#pragma unroll
    for (int c = 0; c < PER; c += 2) *reinterpret_cast<uint32_t *>(p.out_bf16 + at + c) = pack_bf16x2(x[c], x[c + 1]);
  } else if (p.out_bf16) {
#pragma unroll
    for (int c = 0; c < PER; ++c) p.out_bf16[at + c] = float_to_bf16_bits(x[c]);
  }
}

// Whether the tensor-memory form takes these tensors: heads of 128 dims packed densely (a row of heads is a row of the
// tensor map) and 16-byte aligned rows.
static bool tensor_maps_take(const void *q, int dh, int64_t q_row_stride, int64_t q_head_stride, const void *k, const void *v,
                             int64_t n_keys, int64_t kv_row_stride, int64_t kv_head_stride) {
  return dh == 128 && q_head_stride == dh && kv_head_stride == dh && q_row_stride % 8 == 0 && kv_row_stride % 8 == 0 &&
         ((uintptr_t)q % 16) == 0 && ((uintptr_t)k % 16) == 0 && ((uintptr_t)v % 16) == 0 && n_keys >= 1 && n_keys < INT32_MAX;
}

}  // namespace lsa

LSA_API int lsa_band_attend(const uint16_t *q, int64_t R, int Hq, int dh, int64_t q_row_stride,
                            int64_t q_head_stride, const uint16_t *k, const uint16_t *v, int64_t n_keys, int Hkv,
                            int64_t kv_row_stride, int64_t kv_head_stride, int64_t first_position, int window,
                            int sink, float scale, float *out_f32, float *lse, int flags, int32_t *status,
                            void *stream) {
  LSA_REQUIRE(q && k && v && out_f32 && lse, LSA_ERR_NULL);
  LSA_REQUIRE(R >= 0 && Hq >= 1 && Hkv >= 1 && Hq % Hkv == 0 && n_keys >= 0 && first_position >= 0 && window >= 0 &&
                  sink >= 0,
              LSA_ERR_ARGUMENT);
  LSA_REQUIRE(scale > 0.0f, LSA_ERR_ARGUMENT);  // the row maximum is taken before the scale is applied
  LSA_REQUIRE(dh == 64 || dh == 128, LSA_ERR_UNSUPPORTED);
  const int group = Hq / Hkv;
  LSA_REQUIRE(group <= 16 && sink <= lsa::kBandKeys, LSA_ERR_UNSUPPORTED);
  LSA_REQUIRE(kv_row_stride % 8 == 0 && kv_head_stride % 8 == 0 && ((uintptr_t)k % 16) == 0 &&
                  ((uintptr_t)v % 16) == 0 && q_row_stride % 2 == 0 && q_head_stride % 2 == 0 &&
                  ((uintptr_t)q % 4) == 0,
              LSA_ERR_ARGUMENT);
  if (R == 0) return LSA_OK;
  // (a chunk shorter than a tile of rows gains nothing from the tensor-memory form)
  const bool two_term = flags & LSA_BAND_TWO_TERM;
  if (!(flags & LSA_BAND_WARP_MMA) && R >= 128 && first_position + R < INT32_MAX - 256 && ((uintptr_t)out_f32 % 16) == 0 &&
      lsa::tensor_maps_take(q, dh, q_row_stride, q_head_stride, k, v, n_keys, kv_row_stride, kv_head_stride)) {
    lsa::BandTcCall call = {q, k, v, q_row_stride, kv_row_stride, Hkv, {}};
    call.p.out = out_f32, call.p.lse = lse, call.p.status = status;
    call.p.R = (int)R, call.p.n_keys = (int)n_keys, call.p.first_position = (int)first_position;
    call.p.Hq = Hq, call.p.group = group, call.p.window = window, call.p.sink = sink;
    call.p.scale_log2 = scale * 1.4426950408889634f;
    return lsa::launch_band_attend_tc(call, (cudaStream_t)stream);
  }
  lsa::BandParams p;
  p.q = q;
  p.k = k;
  p.v = v;
  p.out = out_f32;
  p.lse = lse;
  p.R = R;
  p.n_keys = n_keys;
  p.first_position = first_position;
  p.q_row_stride = q_row_stride;
  p.q_head_stride = q_head_stride;
  p.kv_row_stride = kv_row_stride;
  p.kv_head_stride = kv_head_stride;
  p.Hq = Hq;
  p.Hkv = Hkv;
  p.group = group;
  p.window = window;
  p.sink = sink;
  p.scale_log2 = scale * 1.4426950408889634f;
  const size_t smem = (size_t)4 * lsa::kBandKeys * dh * 2;
  dim3 grid((unsigned)((R + lsa::kBandRows - 1) / lsa::kBandRows), (unsigned)Hkv, (unsigned)((group + 7) / 8));
  const int threads = (group < 8 ? group : 8) * 32;
  cudaStream_t s = (cudaStream_t)stream;
  auto kernel = dh == 128 ? (two_term ? lsa::band_attend_kernel<128, true> : lsa::band_attend_kernel<128, false>)
                          : (two_term ? lsa::band_attend_kernel<64, true> : lsa::band_attend_kernel<64, false>);
  // 64 KB of tiles a CTA: ask for the largest shared-memory carve-out so that two or three CTAs share an SM
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
      cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared) !=
          cudaSuccess)
    return LSA_ERR_LAUNCH;
  kernel<<<grid, threads, smem, s>>>(p);
  LSA_LAUNCH_CHECK();
  return LSA_OK;
}

LSA_API int lsa_band_round(const float *in, const uint16_t *q, int64_t R, int Hq, int dh, int64_t q_row_stride,
                           int64_t q_head_stride, const uint16_t *k, const uint16_t *v, int64_t n_keys, int Hkv,
                           int64_t kv_row_stride, int64_t kv_head_stride, int64_t first_position, float scale,
                           uint16_t *out_bf16, float *out_f32, void *stream) {
  LSA_REQUIRE(in && q && k && v && (out_bf16 || out_f32), LSA_ERR_NULL);
  LSA_REQUIRE(R >= 0 && Hq >= 1 && Hkv >= 1 && Hq % Hkv == 0 && n_keys >= 0 && first_position >= 0 && scale > 0.0f,
              LSA_ERR_ARGUMENT);
  LSA_REQUIRE(dh == 64 || dh == 128, LSA_ERR_UNSUPPORTED);
  LSA_REQUIRE((R * Hq + 7) / 8 <= INT32_MAX, LSA_ERR_ARGUMENT);
  if (R == 0) return LSA_OK;
  lsa::RoundParams p;
  p.in = in, p.q = q, p.k = k, p.v = v, p.out_bf16 = out_bf16, p.out_f32 = out_f32;
  p.R = R, p.n_keys = n_keys, p.first_position = first_position;
  p.q_row_stride = q_row_stride, p.q_head_stride = q_head_stride;
  p.kv_row_stride = kv_row_stride, p.kv_head_stride = kv_head_stride;
  p.Hq = Hq, p.group = Hq / Hkv;
  p.scale_log2 = scale * 1.4426950408889634f;
  const unsigned grid = (unsigned)((R * Hq + 7) / 8);
  if (dh == 128)
    lsa::band_round_kernel<128><<<grid, 256, 0, (cudaStream_t)stream>>>(p);
  else
    lsa::band_round_kernel<64><<<grid, 256, 0, (cudaStream_t)stream>>>(p);
  LSA_LAUNCH_CHECK();
  return LSA_OK;
}

LSA_API int lsa_dense_attend(const uint16_t *q, int64_t R, int Hq, int dh, int64_t q_row_stride, int64_t q_head_stride,
                             const uint16_t *k, const uint16_t *v, int64_t n_keys, int Hkv, int64_t kv_row_stride,
                             int64_t kv_head_stride, int64_t first_position, const uint32_t *mask, float scale,
                             uint16_t *out_bf16, float *out_f32, int32_t *not_finite, int32_t *status, void *stream) {
  LSA_REQUIRE(q && k && v && (out_bf16 || out_f32) && not_finite, LSA_ERR_NULL);
  LSA_REQUIRE(R >= 0 && Hq >= 1 && Hkv >= 1 && Hq % Hkv == 0 && n_keys >= 0 && first_position >= 0 && scale > 0.0f,
              LSA_ERR_ARGUMENT);
  LSA_REQUIRE(R < INT32_MAX / 2 && first_position < INT32_MAX - 256 - R, LSA_ERR_ARGUMENT);
  LSA_REQUIRE(lsa::tensor_maps_take(q, dh, q_row_stride, q_head_stride, k, v, n_keys, kv_row_stride, kv_head_stride) &&
                  ((uintptr_t)out_bf16 % 16) == 0 && ((uintptr_t)out_f32 % 16) == 0 && ((uintptr_t)mask % 16) == 0,
              LSA_ERR_UNSUPPORTED);
  if (R == 0) return LSA_OK;
  cudaStream_t s = (cudaStream_t)stream;
  if (cudaMemsetAsync(not_finite, 0, 4, s) != cudaSuccess) return LSA_ERR_LAUNCH;
  lsa::BandTcCall call = {q, k, v, q_row_stride, kv_row_stride, Hkv, {}};
  call.p.out = out_f32, call.p.out_bf16 = out_bf16, call.p.not_finite = not_finite, call.p.status = status;
  call.p.mask = reinterpret_cast<const uint4 *>(mask);
  call.p.R = (int)R, call.p.n_keys = (int)n_keys, call.p.first_position = (int)first_position;
  call.p.Hq = Hq, call.p.group = Hq / Hkv, call.p.window = (int)(first_position + R), call.p.sink = 0;
  call.p.scale_log2 = scale * 1.4426950408889634f;
  const int rc = lsa::launch_band_attend_tc(call, s);
  if (rc != LSA_OK) return rc;
  lsa::RoundParams p = {};
  p.q = q, p.k = k, p.v = v, p.out_bf16 = out_bf16, p.out_f32 = out_f32;
  p.R = R, p.n_keys = n_keys, p.first_position = first_position;
  p.q_row_stride = q_row_stride, p.q_head_stride = q_head_stride;
  p.kv_row_stride = kv_row_stride, p.kv_head_stride = kv_head_stride;
  p.Hq = Hq, p.group = Hq / Hkv;
  p.scale_log2 = scale * 1.4426950408889634f;
  const int64_t ctas = (R * Hq + lsa::kAgainWarps - 1) / lsa::kAgainWarps, most = 4 * (int64_t)lsa::sm_count();
  lsa::dense_repair_kernel<<<(unsigned)(ctas < most ? ctas : most), lsa::kAgainWarps * 32, 0, s>>>(p, mask, not_finite);
  LSA_LAUNCH_CHECK();
  return LSA_OK;
}
