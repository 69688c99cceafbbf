// Which keys a row's list names, as one bit a key: what the listed form of the dense read masks with. The list is that of
// lsa_expand - members best bucket first up to the row's top-k, the window, the sinks - without its order.
//
// A warp a row, eight rows a CTA. Buckets of 16 places are a lane each, wider ones several. A lane takes its places twice - how
// many count, then, once the counts before it are summed, its share of the top-k - and sets their bits in the row's words in
// shared memory: sixteen places are held in registers from one read where they lie 16 bytes at a time, others are walked. A pool's
// keys are neighbours, so four of them are one step and a lane gathers a word's bits before it adds them. The eight rows' words
// leave together, 128 bytes a key tile. What bounds it is the warps' own instructions (20,096 rows of up to 4,096 keys out of 1,024
// picks of 16 places, half full: 303 us, where expansion into lists takes 696; a list and a walk of it would write and read four
// bytes a key in place of a bit).
#include "common.cuh"

namespace lsa {

constexpr int kBitsRows = 8, kBitsQuads = 4;
constexpr size_t kBitsShared = 200 * 1024;

struct ListBitsParams {
  const int32_t *picked, *members, *row_top_p, *row_top_k;
  const int64_t *positions;
  uint4 *mask;
  int32_t *status;
  int64_t R, m, n_keys;
  int top_p, cap, top_k, sink, window, tiles;
  int lanes, places;  // lanes a pick, and places of its bucket a lane
  bool quads;         // members may be read 16 bytes at a time
};

__global__ void __launch_bounds__(kBitsRows * 32) list_bits_kernel(ListBitsParams p) {
  extern __shared__ __align__(16) uint32_t words_s[];
  const int warp = threadIdx.x >> 5, lane = lane_id();
  const int row_words = p.tiles * 4;
  const int64_t r = (int64_t)blockIdx.x * kBitsRows + warp;
  uint32_t *words = words_s + warp * row_words;
  for (int i = lane; i < row_words; i += 32) words[i] = 0u;
  __syncwarp();
  if (r < p.R) {
    const int64_t pos = p.positions[r];
    const int row_p = p.row_top_p ? max(0, min(p.row_top_p[r], p.top_p)) : p.top_p;
    const int row_k = p.row_top_k ? max(0, min(p.row_top_k[r], p.top_k)) : p.top_k;
    const int64_t window_start = max((int64_t)0, pos + 1 - p.window);
    const int64_t key_end = min(p.n_keys, (int64_t)p.tiles * 128);
    int counted = 0, bad = 0;
    const int in_step = 32 / p.lanes, first = lane % p.lanes * p.places, places = min(p.places, p.cap - first);
    const bool sixteen = p.quads && p.places == 4 * kBitsQuads && p.cap % p.places == 0;  // (the same in every lane)
    int i0 = 0;
    for (; i0 < row_p && counted < row_k; i0 += in_step) {
      const int i = i0 + lane / p.lanes;
      int64_t bucket = i < row_p ? p.picked[r * p.top_p + i] : -1;
      if (bucket >= p.m) {
        bucket = -1;
        bad += first == 0;
      }
      const int32_t *row = p.members + (bucket >= 0 ? bucket * p.cap + first : 0);
      // the members at this lane's places in order, until `see` has had enough
      auto walk = [&](auto see) {
        if (bucket < 0) return;
        if (p.quads) {
          const int4 *row4 = reinterpret_cast<const int4 *>(row);
          for (int j = 0; j < places / 4; ++j) {
            const int4 ids = row4[j];
            if (!see(ids.x) || !see(ids.y) || !see(ids.z) || !see(ids.w)) return;
          }
        } else {
          for (int j = 0; j < places; ++j)
            if (!see(row[j])) return;
        }
      };
      // (a row of members ends in padding, whose ids are under every sink)
      const uint32_t span = window_start > p.sink ? (uint32_t)(window_start - p.sink) : 0u;
      auto counts = [&](int32_t id) { return (uint32_t)id - (uint32_t)p.sink < span && id >= 0; };
      int4 held[kBitsQuads];  // sixteen places a lane, read once where they lie 16 bytes at a time
      int n = 0;
      if (sixteen) {
        const int4 *row4 = reinterpret_cast<const int4 *>(row);
        const bool any = bucket >= 0 && places > 0;  // (the lanes are a power of two: 112 places are seven lanes', and the eighth has none)
#pragma unroll
        for (int j = 0; j < kBitsQuads; ++j) held[j] = any ? row4[j] : make_int4(-1, -1, -1, -1);
#pragma unroll
        for (int j = 0; j < kBitsQuads; ++j)
          n += (counts(held[j].x) ? 1 : 0) + (counts(held[j].y) ? 1 : 0) + (counts(held[j].z) ? 1 : 0) + (counts(held[j].w) ? 1 : 0);
      } else {
        walk([&](int32_t id) {
          n += counts(id);
          return id >= 0;
        });
      }
      int incl = n;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += up;
      }
      int left = min(n, row_k - (counted + incl - n));
      if (left > 0) {
        int at = 0;
        uint32_t bits = 0u;
        auto add = [&](int32_t id) {
          if (!counts(id)) return true;
          if (id < key_end) {
            if (id >> 5 != at) {
              if (bits) atomicOr(&words[at], bits);
              at = id >> 5, bits = 0u;
            }
            bits |= 1u << (id & 31);
          }
          return --left > 0;
        };
        if (sixteen) {
#pragma unroll
          for (int j = 0; j < kBitsQuads; ++j) {
            // (four keys that all count and are neighbours in a word, as a pool's are: one step)
            const int4 v = held[j];
            const bool run = left >= 4 && v.w == v.x + 3 && v.y == v.x + 1 && v.z == v.x + 2 && (v.x & 31) <= 28 && counts(v.x) &&
                             counts(v.w) && v.w < key_end;
            if (run) {
              if (v.x >> 5 != at) {
                if (bits) atomicOr(&words[at], bits);
                at = v.x >> 5, bits = 0u;
              }
              bits |= 0xFu << (v.x & 31);
              left -= 4;
            } else if (left > 0) {
              if (add(v.x) && add(v.y) && add(v.z)) add(v.w);
            }
          }
        } else {
          walk(add);
        }
        if (bits) atomicOr(&words[at], bits);
      }
      counted += __shfl_sync(0xffffffffu, incl, 31);
    }
    // (picks past the cut add no key, but those outside the table are told of as well)
    for (int i = i0 + lane; i < row_p; i += 32) bad += p.picked[r * p.top_p + i] >= p.m;
    __syncwarp();
    // the window, and the sinks that lie before it
    const int64_t end = min(pos + 1, key_end), sinks = min((int64_t)p.sink, min(window_start, end));
    auto below = [](int64_t x) { return x >= 32 ? 0xffffffffu : (x <= 0 ? 0u : (1u << (int)x) - 1u); };
    for (int i = lane; i < row_words; i += 32) {
      const int64_t key = (int64_t)i * 32;
      words[i] |= (below(end - key) & ~below(window_start - key)) | below(sinks - key);
    }
    bad = warp_sum_int(bad);
    if (lane == 0 && bad && p.status) atomicAdd(p.status, bad);
  }
  __syncthreads();
  const int64_t r0 = (int64_t)blockIdx.x * kBitsRows;
  for (int i = threadIdx.x; i < p.tiles * kBitsRows; i += kBitsRows * 32) {
    const int tile = i / kBitsRows, at = i - tile * kBitsRows;
    if (r0 + at < p.R)
      p.mask[(int64_t)tile * p.R + r0 + at] = *reinterpret_cast<const uint4 *>(words_s + at * row_words + tile * 4);
  }
}

}  // namespace lsa

LSA_API int lsa_list_bits(const int32_t *picked, int64_t R, int top_p, const int64_t *positions, const int32_t *members,
                          int64_t m, int cap, const int32_t *row_top_p, const int32_t *row_top_k, int top_k, int sink,
                          int window, int64_t n_keys, int tiles, uint32_t *mask, int32_t *status, void *stream) {
  LSA_REQUIRE(positions && mask && (top_p == 0 || (picked && (members || m == 0))), LSA_ERR_NULL);
  LSA_REQUIRE(R >= 0 && top_p >= 0 && m >= 0 && cap >= 1 && top_k >= 0 && sink >= 0 && window >= 0 && n_keys >= 0 && tiles >= 1,
              LSA_ERR_ARGUMENT);
  const size_t smem = (size_t)tiles * 16 * lsa::kBitsRows;
  LSA_REQUIRE(smem <= lsa::kBitsShared && ((uintptr_t)mask % 16) == 0, LSA_ERR_UNSUPPORTED);
  LSA_REQUIRE((R + lsa::kBitsRows - 1) / lsa::kBitsRows <= INT32_MAX, LSA_ERR_ARGUMENT);
  if (R == 0) return LSA_OK;
  int lanes = 1;
  while (lanes < 32 && cap > 16 * lanes) lanes *= 2;
  const int places = ((cap + lanes - 1) / lanes + 3) & ~3;
  lsa::ListBitsParams p = {picked, members, row_top_p, row_top_k, positions, reinterpret_cast<uint4 *>(mask), status, R, m,
                           n_keys, top_p, cap, top_k, sink, window, tiles, lanes, places,
                           cap % 4 == 0 && ((uintptr_t)members % 16) == 0};
  if (!lsa::allow_shared(lsa::list_bits_kernel, lsa::kBitsShared)) return LSA_ERR_LAUNCH;
  lsa::list_bits_kernel<<<(unsigned)((R + lsa::kBitsRows - 1) / lsa::kBitsRows), lsa::kBitsRows * 32, smem,
                          (cudaStream_t)stream>>>(p);
  LSA_LAUNCH_CHECK();
  return LSA_OK;
}
