// The attend pass of the bucket-major attention on the fifth-generation tensor cores.
//
// A CTA owns (bucket, KV head, segment of up to 256 (row, pick) pairs). The M = 128 rows of a tile are (pair, query
// head of the KV head's group) couples, the heads of a pair next to one another, so a ragged segment of n pairs
// costs ceil(n * group / 128) tiles and not `group` of them. A row of S and of O lives in one lane of tensor memory
// and the thread that owns the row does its softmax without talking to anyone:
//
//   S [128 x keys]  = Q [128 x 128] . K^T           tcgen05.mma, A = the tile's query rows, B = the bucket's keys,
//                                                   both K-major planes of 64 dims with the 128-byte swizzle
//   P               = exp2(S - rowmax) on the row's key range, bf16, written back to shared memory (divided by the
//                     row's sum first where a thread can hold the whole row: buckets of up to 64 keys)
//   O [128 x 128]   = P [128 x keys] . V            A = P (K-major), B = the bucket's values AS STORED
//                                                   ([key][dim] planes: an MN-major operand)
//
// Two warpgroups, each with tiles of its own (every other tile of the segment), its own query buffer and its own 128
// columns of tensor memory (O takes the columns of S, which has been read by then). A warp copies, multiplies and writes
// out ITS 32 rows, so between the hand-overs to the tensor cores nothing waits for another warp; a
// warpgroup's first warp issues its products. Two CTAs share an SM (buckets of up to 64 keys), so four tiles are under
// way on it and fill one another's waits. What bounds it is the instruction stream around the products and the chain
// copy - product - softmax - product - copy of a tile: 0.85 G warp instructions a launch of 8,192 rows x 64 picks x 40 heads,
// issued on 41 % of the cycles. (With both warpgroups on ONE tile, two threads a row, swapping maxima and sums and waiting
// for one another six times a tile, it was 1.2 G; a 131,072-token prompt spent 41.1 ms here, and 35.3 after that step.) Buckets of 65
// to 128 members take twice the shared memory, so one CTA an SM, and a thread reads its row of S twice.
// Their partial outputs are fp32: the gather, which such buckets have too, holds a row's sums in fp32 from its first key to
// its last, and rounded partials were further from the sums in 64 bits than it is (a 16,384-token prompt of 64-key buckets,
// 2-norm of the bf16 output's error over the output's: gather 1.6619e-3, bf16 partials 1.6624e-3, fp32 partials 1.6587e-3; the
// whole prefill 2.21, 1.23 and 1.40 ms).
//
// Shared-memory operands are written by ordinary and asynchronous copies (the generic proxy), so a proxy fence stands
// before every hand-over to the tensor cores. Every wait on an mbarrier is bounded; a wait that gives up raises the
// CTA's abort flag, the CTA skips its remaining work (but none of its barriers), frees its tensor memory and leaves.
#include "bucket_attend.cuh"
#include "mma.cuh"
#include "umma.cuh"

namespace lsa {

constexpr int kTcThreads = 256;
constexpr int kTcRows = 128;                    // rows of a tile: a warpgroup's threads
constexpr int kTcQPlane = kTcRows * 128;        // a plane (64 dims) of the query tile, of P (64 keys) or of finished rows
constexpr int kTcTmemCols = 256;                // 128 columns a warpgroup: S, then O
static_assert(kBktSegmentTc == kTcThreads, "a thread a pair of the segment");

// Shared memory: K and V (2 planes of 64 dims each), then a query buffer of two planes a warpgroup. P takes the query
// buffer's planes (the first product is over when P is written), and the finished rows of O are staged in the whole of it
// (the second product is over by then).
template <int KEYS>
constexpr int tc_smem() {
  return 4 * KEYS * 128 + 2 * 2 * kTcQPlane + 1024;  // + room to align the base to 1,024 bytes
}

__device__ __forceinline__ void proxy_fence() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

// KEYS: members a bucket may hold, 64 or 128.
template <int DH, int KEYS>
__global__ void __launch_bounds__(kTcThreads, KEYS == 64 ? 2 : 1) bucket_attend_tc_kernel(BucketParams p) {
  static_assert(DH == 128, "two planes of 64 dims");
  constexpr int kPlane = KEYS * 128;           // a plane of KEYS rows x 64 dims
  constexpr int kKOff = 0, kVOff = 2 * kPlane, kQOff = 4 * kPlane;
  constexpr int kWords = KEYS / 32;
  constexpr bool kHeld = KEYS == 64;           // a thread holds its whole row of S, and partials leave in bf16
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  __shared__ int32_t ids_s[KEYS];
  __shared__ int32_t pairs_s[kBktSegmentTc];   // the segment's pairs, -1 past its end
  __shared__ int32_t qrows_s[kBktSegmentTc];   // their query rows
  __shared__ int32_t hi_s[kBktSegmentTc];      // members of the bucket they read
  __shared__ int64_t src_s[2][kTcRows];        // where the query rows of a warpgroup's tile start in q, -1 past the end
  __shared__ __align__(8) uint64_t bars[6];
  __shared__ uint32_t tmem_base_s;
  __shared__ volatile int abort_s;
  __shared__ uint32_t valid_s[kWords];         // which members of the bucket name a row of the cache

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int seg = blockIdx.x;
  // (the table holds a slot for every CTA of the grid: the segment is asked for beside the count, not after it)
  const int4 info = p.segments[seg];
  if (seg >= p.seg_offsets[p.m]) return;
  const int64_t bucket = info.x;
  const int first = info.y, n_pairs = info.z;
  const int n_rows = n_pairs * p.group;
  const int n_tiles = (n_rows + kTcRows - 1) / kTcRows;
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const int wg = warp >> 2;                  // the warpgroup
  const int quarter = warp & 3;              // the 32 tensor-memory lanes (and tile rows) this warp has
  const int row = quarter * 32 + lane;       // the tile row (= tensor-memory lane)
  // of the warpgroup - bar_w: its threads tell its issuing lane that operands are in place (queries, then P, of every
  // tile); bar_s / bar_o: a product has finished
  const uint32_t bar_w = smem_u32(&bars[wg]), bar_s = smem_u32(&bars[2 + wg]), bar_o = smem_u32(&bars[4 + wg]);

  if (tid == 0) {
    for (int i = 0; i < 6; ++i) mbar_init(smem_u32(&bars[i]), i < 2 ? kTcRows : 1);
    abort_s = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)),
                 "r"(kTcTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
  }
  for (int i = tid; i < KEYS; i += kTcThreads) ids_s[i] = i < p.cap ? p.members[bucket * p.cap + i] : LSA_PAD;
  // The segment's pairs, fetched beside the member ids (one round of loads for both). The starts pass has counted the
  // keys a pair takes; its run of members starts where the sinks end, which is added once the ids are in.
  {
    int32_t pair = -1, take = 0;
    if (tid < n_pairs) {
      pair = p.order[first + tid];
      take = p.order_takes[first + tid];
    }
    pairs_s[tid] = pair, qrows_s[tid] = pair >= 0 ? pair / p.top_p : 0, hi_s[tid] = take;
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_base_s + wg * DH;
  const uint32_t buf = base + kQOff + wg * 2 * kTcQPlane;  // the warpgroup's query buffer

  // members of the bucket: the ids before the first pad; and which of them name a row of the cache handed in (a key
  // outside it is staged as zeros and masked out of the softmax, as the row-by-row read skips such ids)
  int n_members = 0;
  bool all_valid = true, ended = false;
#pragma unroll
  for (int w = 0; w < kWords; ++w) {
    const int32_t id = ids_s[32 * w + lane];
    const unsigned some = __ballot_sync(0xffffffffu, id >= 0), valid = __ballot_sync(0xffffffffu, id >= 0 && id < p.slots);
    if (!ended) n_members += some != 0xffffffffu ? __ffs(~some) - 1 : 32;
    ended = ended || some != 0xffffffffu;
    all_valid = all_valid && valid == some;
    if (tid == 0) valid_s[w] = valid;
  }
  n_members = min(n_members, p.cap);
  // (the words stay in shared memory and only a flag in a register: every member is in the cache as a rule)
  auto valid_byte = [&](int c0) { return all_valid ? 0xFFu : (valid_s[c0 >> 5] >> (c0 & 31)) & 0xFFu; };
  const int n_keys = max(16, (n_members + 15) & ~15);  // the N of S and the K of O: whole 16-key steps
  int lo_key = 0;
  {
    int hi = n_members;
    while (lo_key < hi) {
      const int mid = (lo_key + hi) >> 1;
      if (ids_s[mid] < p.sink) lo_key = mid + 1; else hi = mid;
    }
  }
  // The bucket's keys and values of a KV head: chunk c of member j goes to plane c / 8, row j, 16-byte slot
  // (c % 8) ^ (j % 8) - the layout a tensor-map copy with the 128-byte swizzle would write.
  auto stage_kv = [&](int h) {
    const uint16_t *k_head = p.k + (int64_t)h * p.kv_head_stride, *v_head = p.v + (int64_t)h * p.kv_head_stride;
#pragma unroll 2
    for (int e = tid; e < n_keys * 16; e += kTcThreads) {
      const int r = e >> 4, chunk = e & 15;
      const int32_t id = ids_s[r];
      const bool ok = id >= 0 && id < p.slots;
      const int64_t off = ok ? (int64_t)id * p.kv_row_stride + chunk * 8 : 0;
      const uint32_t dst = (chunk >> 3) * kPlane + r * 128 + (((chunk & 7) ^ (r & 7)) << 4);
      cp_async_16(base + kKOff + dst, k_head + off, ok ? 16 : 0);
      cp_async_16(base + kVOff + dst, v_head + off, ok ? 16 : 0);
    }
    cp_async_commit();
  };
  const uint32_t group_inverse = (65536u + (uint32_t)p.group - 1) / (uint32_t)p.group;  // flat / group, exact here
  int hi_key = 0;       // of this thread's row: the end of its key range,
  int32_t slot = -1;    // and the slot of the partial outputs it fills (the caller has checked that slots fit 31 bits)
  auto list_rows = [&](int h, int tile) {
    const int flat = tile * kTcRows + row;
    const bool ok = flat < n_rows;
    const int pl = ok ? (int)((uint32_t)flat * group_inverse >> 16) : 0;
    const int head = h * p.group + (flat - pl * p.group);
    src_s[wg][row] = ok ? (int64_t)qrows_s[pl] * p.q_row_stride + (int64_t)head * p.q_head_stride : -1;
    slot = ok ? pairs_s[pl] * p.Hq + head : -1;
    hi_key = ok ? lo_key + hi_s[pl] : 0;
    __syncwarp();
  };
  // The warp's query rows of a tile: half a warp copies a row of 256 bytes, in the layout of the keys.
  const int chunk = lane & 15;
  const uint32_t lane_at = (chunk >> 3) * kTcQPlane + quarter * 32 * 128;
  auto gather_q = [&] {
#pragma unroll 8
    for (int j = 0; j < 16; ++j) {
      const int r = 2 * j + (lane >> 4);  // of the warp's 32
      const int64_t from = src_s[wg][quarter * 32 + r];
      cp_async_16(buf + lane_at + r * 128 + (((chunk & 7) ^ (r & 7)) << 4), p.q + (from >= 0 ? from + chunk * 8 : 0),
                  from >= 0 ? 16 : 0);
    }
    cp_async_commit();
  };
  // The issuing lane's turn (the whole warp waits so that its lanes stay together): false once the CTA has given up.
  auto my_turn = [&](uint32_t parity) {
    if (__all_sync(0xffffffffu, !abort_s && mbar_wait(bar_w, parity))) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      return true;
    }
    abort_s = 1;
    return false;
  };

  const uint32_t lane_addr = tmem + ((uint32_t)(quarter * 32) << 16);
  // One KV head after another: the segment, the bucket's members and the pairs are fetched once, three dependent rounds
  // of loads that a CTA a head paid before each head's first product (131,072 tokens of 40 heads over 8: 35.3 -> 33.8 ms).
  int n = 0;  // tiles this warpgroup has had
  const int end_head = (blockIdx.y + 1) * p.heads_a_cta;
  for (int h = blockIdx.y * p.heads_a_cta; h < end_head; ++h) {
    stage_kv(h);
    if (wg < n_tiles) {
      list_rows(h, wg);
      gather_q();
    }
    cp_async_wait<0>();
    proxy_fence();
    __syncthreads();  // K and V are in place (a warpgroup without tiles has copied its share too)
    for (int tile = wg; tile < n_tiles; tile += 2, ++n) {
      const uint32_t parity = n & 1;
      if (tile > wg) {
        cp_async_wait<0>();
        proxy_fence();
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      mbar_arrive(bar_w);  // this thread's part of the tile's queries is in place, and it has read its row of the last O
      if (quarter == 0 && my_turn(0) && elect_one()) {  // S = Q K^T: 16 dims are 32 bytes further inside the swizzle atom
        const uint64_t q_desc = smem_desc_sw128(buf), k_desc = smem_desc_sw128(base + kKOff);
#pragma unroll
        for (int plane = 0; plane < 2; ++plane)
#pragma unroll
          for (int s = 0; s < 4; ++s)
            umma_bf16(tmem, q_desc + (plane * kTcQPlane >> 4) + 2 * s, k_desc + (plane * kPlane >> 4) + 2 * s,
                      umma_idesc(n_keys), (plane | s) != 0);
        umma_commit(bar_s);
      }
      __syncwarp();
      // A group of 8 keys that lies inside the key range of every row of the warp needs no masks: most do.
      const int hi_min = __reduce_min_sync(0xffffffffu, hi_key);
      auto whole = [&](int c0) { return c0 >= lo_key && c0 + 8 <= hi_min && valid_byte(c0) == 0xFFu; };
      // ---- softmax of the row: P is the A operand of the second product. (One decision a warp on a wait: the
      // tensor-memory loads are warp-wide instructions.)
      bool go = __all_sync(0xffffffffu, !abort_s && mbar_wait(bar_s, parity));
      if (!go) abort_s = 1;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      uint32_t sv[kHeld ? kWords : 1][32];
      // keys 32 c .. 32 c + 31 of the row, the masked ones at -inf
      auto load_keys = [&](int c, uint32_t (&v)[32]) {
        if (go) tmem_load_32(lane_addr + 32 * c, v);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int c0 = 32 * c + 8 * j;
          if (c0 >= n_keys || whole(c0)) continue;
          const uint32_t vb = valid_byte(c0);
#pragma unroll
          for (int i = 0; i < 8; ++i) {  // (bitwise logic and selects: branches here would diverge lane by lane)
            const bool ok = (c0 + i >= lo_key) & (c0 + i < hi_key) & (bool)((vb >> i) & 1u);
            v[8 * j + i] = ok ? v[8 * j + i] : 0xFF800000u;
          }
        }
      };
      // (four running maxima, and four running sums below: one chain of 64 dependent operations is what a thread with few
      // warps beside it waits on)
      float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int c = 0; c < kWords; ++c) {
        if (32 * c >= n_keys) continue;
        uint32_t (&v)[32] = sv[kHeld ? c : 0];
        load_keys(c, v);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (32 * c + 8 * j >= n_keys) continue;
#pragma unroll
          for (int i = 0; i < 8; ++i) mx4[i & 3] = fmaxf(mx4[i & 3], __uint_as_float(v[8 * j + i]));
        }
      }
      const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
      const float m_row = mx == -INFINITY ? 0.0f : mx * p.scale_log2;  // (finite, so that a masked key gives exp2(-inf) = 0)
      float l4[4] = {0.0f, 0.0f, 0.0f, 0.0f};
      auto exponentials = [&](int c, uint32_t (&v)[32]) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (32 * c + 8 * j >= n_keys) continue;
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const float e = fast_exp2(fmaf(__uint_as_float(v[8 * j + i]), p.scale_log2, -m_row));
            l4[i & 3] += e;
            v[8 * j + i] = __float_as_uint(e);
          }
        }
      };
      // 16-byte slot (key / 8 % 8) ^ (row % 8) of the row, in the plane of the key's 64
      auto store_p = [&](int c, uint32_t (&v)[32], float by) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int c8 = 4 * c + j;
          if (8 * c8 >= n_keys) continue;
          uint32_t w[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float a = __uint_as_float(v[8 * j + 2 * i]), b = __uint_as_float(v[8 * j + 2 * i + 1]);
            w[i] = kHeld ? pack_bf16x2(a * by, b * by) : pack_bf16x2(a, b);
          }
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(buf + (c8 >> 3) * kTcQPlane + row * 128 +
                                                                         (((c8 & 7) ^ (row & 7)) << 4)),
                       "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3])
                       : "memory");
        }
      };
#pragma unroll
      for (int c = 0; c < kWords; ++c) {
        if (32 * c >= n_keys) continue;
        uint32_t (&v)[32] = sv[kHeld ? c : 0];
        if constexpr (!kHeld) load_keys(c, v);
        exponentials(c, v);
        if constexpr (!kHeld) store_p(c, v, 1.0f);
      }
      const float l_row = (l4[0] + l4[1]) + (l4[2] + l4[3]);
      const float inv = (kHeld ? l_row > 0.0f : l_row != 0.0f) ? 1.0f / l_row : 0.0f;
      if constexpr (kHeld) {
#pragma unroll
        for (int c = 0; c < kWords; ++c)
          if (32 * c < n_keys) store_p(c, sv[c], inv);
      }
      float lse = l_row > 0.0f ? (m_row + log2f(l_row)) * 0.6931471805599453f : -INFINITY;
      // (a score that is not a number is carried out of a wide bucket, as the gather carries it: infinity is the
      // log-sum-exp that the merge cannot leave out)
      if (!kHeld && isnan(l_row)) lse = INFINITY;
      if (go && slot >= 0) p.part_lse[slot] = lse;
      proxy_fence();
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      mbar_arrive(bar_w);
      if (quarter == 0 && my_turn(1) && elect_one()) {  // O = P V: 16 keys are 32 bytes along P's rows, 2,048 down V's planes
        const uint64_t p_desc = smem_desc_sw128(buf), v_desc = smem_desc_mn_sw128(base + kVOff, kPlane);
#pragma unroll
        for (int s = 0; s < KEYS / 16; ++s)
          if (16 * s < n_keys)
            umma_bf16(tmem, p_desc + ((s >> 2) * kTcQPlane >> 4) + 2 * (s & 3), v_desc + (s * 2048 >> 4), umma_idesc(DH, true),
                      s != 0);
        umma_commit(bar_o);
      }
      __syncwarp();
      // ---- O of the tile: out of tensor memory into the tile's (spent) query buffer, then out in whole rows
      go = __all_sync(0xffffffffu, !abort_s && mbar_wait(bar_o, parity));
      if (!go) abort_s = 1;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      // 16-byte piece `at` (of 16) of the row: a plane of the buffer holds eight, laid out as the query rows were, so a
      // warp's rows stay inside the bytes that the warp itself fills again
      auto stage_piece = [&](int at, uint32_t w0, uint32_t w1, uint32_t w2, uint32_t w3) {
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(buf + (at >> 3) * kTcQPlane + row * 128 +
                                                                       (((at & 7) ^ (row & 7)) << 4)),
                     "r"(w0), "r"(w1), "r"(w2), "r"(w3)
                     : "memory");
      };
      // The warp's staged rows, half a warp a row, to where its slots begin (16-byte pieces a slot: `pitch`). Eight rows' pieces
      // are on their way out of shared memory together: one after another, each behind a branch on its slot, this was a fifth of a
      // tile's time.
      auto write_out = [&](uint4 *to_slot_0, int pitch) {
#pragma unroll
        for (int j0 = 0; j0 < 16; j0 += 8) {
          uint4 piece[8];
          int32_t to[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const int r = 2 * (j0 + j) + (lane >> 4);
            to[j] = __shfl_sync(0xffffffffu, slot, r);
            asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                         : "=r"(piece[j].x), "=r"(piece[j].y), "=r"(piece[j].z), "=r"(piece[j].w)
                         : "r"(buf + lane_at + r * 128 + (((chunk & 7) ^ (r & 7)) << 4)));
          }
#pragma unroll
          for (int j = 0; j < 8; ++j)
            if (to[j] >= 0) to_slot_0[(int64_t)to[j] * pitch + chunk] = piece[j];
        }
      };
      uint4 *parts = reinterpret_cast<uint4 *>(p.part_out);
#pragma unroll
      for (int half = 0; half < 2; ++half) {  // 64 columns: a plane of bf16, or both planes of fp32
        if (go) {
          uint32_t r[2][32];
          tmem_load_32(lane_addr + half * 64, r[0]);
          tmem_load_32(lane_addr + half * 64 + 32, r[1]);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              uint32_t (&v)[32] = r[c];
              if constexpr (kHeld) {
                uint32_t w[4];
#pragma unroll
                for (int k = 0; k < 4; ++k)
                  w[k] = pack_bf16x2(__uint_as_float(v[8 * i + 2 * k]), __uint_as_float(v[8 * i + 2 * k + 1]));
                stage_piece(half * 8 + c * 4 + i, w[0], w[1], w[2], w[3]);
              } else {
                uint32_t w[8];
#pragma unroll
                for (int k = 0; k < 8; ++k) w[k] = __float_as_uint(__uint_as_float(v[8 * i + k]) * inv);
                stage_piece(c * 8 + 2 * i, w[0], w[1], w[2], w[3]);
                stage_piece(c * 8 + 2 * i + 1, w[4], w[5], w[6], w[7]);
              }
            }
        }
        if (kHeld && half == 0) continue;  // (both halves of a bf16 row leave together)
        __syncwarp();  // the warp's rows are staged
        if (go) write_out(kHeld ? parts : parts + half * 16, kHeld ? DH / 8 : DH / 4);
        __syncwarp();  // and have been read out
      }
      if (tile + 2 < n_tiles) {
        list_rows(h, tile + 2);
        gather_q();
      }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();  // every product over this head's keys and values is over
  }
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base_s), "r"(kTcTmemCols));
  }
  // A CTA that gave up leaves stale partials behind: the status word tells the host that the call's output is void.
  if (tid == 0 && abort_s && p.status) atomicAdd(p.status, 1);
}

template <int KEYS>
static int launch_tc(const BucketParams &p, int64_t segment_bound, cudaStream_t stream) {
  auto kernel = bucket_attend_tc_kernel<128, KEYS>;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, tc_smem<KEYS>()) != cudaSuccess)
    return LSA_ERR_LAUNCH;
  const dim3 grid((unsigned)segment_bound, (unsigned)(p.Hkv / p.heads_a_cta));
  kernel<<<grid, kTcThreads, tc_smem<KEYS>(), stream>>>(p);
  LSA_LAUNCH_CHECK();
  return LSA_OK;
}

int launch_bucket_attend_tc(const BucketParams &params, int64_t segment_bound, cudaStream_t stream) {
  BucketParams p = params;
  // As many heads a CTA as leave eight waves of two CTAs an SM, counting the segments that full ones would make.
  const int64_t segments = p.R * p.top_p / p.segment;
  p.heads_a_cta = 1;
  while (p.Hkv % (2 * p.heads_a_cta) == 0 && segments * (p.Hkv / (2 * p.heads_a_cta)) >= 16 * (int64_t)sm_count())
    p.heads_a_cta *= 2;
  return p.cap <= 64 ? launch_tc<64>(p, segment_bound, stream) : launch_tc<128>(p, segment_bound, stream);
}

}  // namespace lsa
