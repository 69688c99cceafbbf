// Dense attention of consecutive query rows on the fifth-generation tensor cores: the window and the sinks of a prefill
// (a band), every key up to a row's own (a causal read), or the keys a row's list names out of those (a listed read, the
// lists handed in as one bit a key).
//
// A CTA owns two tiles of 128 consecutive query rows of ONE query head and walks the keys they see once, in tiles of 128.
// The rows are the M = 128 side of both products, so a row of S and of O lives in one lane of tensor memory. The probabilities
// go back into tensor memory over the scores they came from, as bf16 and what bf16 left of them, and are the A operand of the
// second product from there:
//
//   columns   0-127 / 128-255   S of tile 0 / 1, then P: of each 32 keys 16 columns of first terms and 16 of second ones
//   columns 256-383 / 384-511   O of tile 0 / 1
//
//   warp 0       one lane streams key and value tiles with tensor-map copies (128-byte swizzle) through a ring of four
//   warp 1       tensor-memory allocation; it issues, for tile 0 and tile 1 in turn, O += P V of the last keys and
//                S = Q K^T of the next, so the products of one tile run while the other is in its softmax
//   warps 2-17   the softmax, two threads a row: 64 of a step's 128 keys each
//
// A row's exponents are taken against a running maximum that follows the true one lazily: it moves, and O and the sum so far
// are scaled, only when a tile holds a score 2^8 times as heavy. (O is complete then: the issuing warp's commit of S covers
// every product before it. And a product adds to all 128 columns of O, of which a row's two threads scale 64 each: none is
// issued until the threads of BOTH halves have arrived with their P, and with it their columns scaled.) Probabilities are 2^8 at most, and their two terms hold them to 2^-17 of themselves, so what the
// reference point is does not show.
//
// What bounds it is the chain of a step, some 2,600 cycles a tile: 1,536 of products (the two terms of P cost a second one) that
// alternate with the other tile's, 1,900 of softmax that four warps a scheduler share, and the hand-overs, the wait between a
// tile's P V and the S that is written over its P among them. The tensor pipe is active 59 % of the time. 16,384 causal rows of 40 heads over 8: 3.39 ms, 811 TFLOP/s of useful work and 1,217 with the second term counted (3.24
// without the wait; 5.61 when the keys were walked twice, maxima then sums, with P in shared memory and one tile a CTA); a masked
// read of the same rows 3.65. 8,192 rows of a band of 1,024 keys 0.40 ms (0.53): a CTA's ten steps stand beside its start and its
// end. Tried: S in two buffers of 64 keys a tile (drains the pipe), a thread a row (a softmax of 3,400 cycles a step).
//
// Every wait on an mbarrier is bounded; a wait that gives up raises the CTA's abort flag and the status word, the
// roles drain, the tensor memory is freed and the CTA leaves.
#include "band_attend.cuh"
#include "common.cuh"
#include "mma.cuh"
#include "umma.cuh"

namespace lsa {

constexpr int kBtRows = 128;
constexpr int kBtTiles = 2;                          // tiles of rows a CTA
constexpr int kBtKeys = 128;                         // keys a tile: N of S, K of O
constexpr int kBtThreads = 576;                      // the copying warp, the issuing warp and sixteen of softmax
constexpr int kBtStages = 4;                         // ring slots, each a key or a value tile
constexpr int kBtPlane = kBtKeys * 128;              // 128 keys (or rows) x 64 dims of bf16
constexpr int kBtSlot = 2 * kBtPlane;
constexpr int kBtSmem = kBtTiles * 2 * kBtPlane + kBtStages * kBtSlot + 1024;
constexpr int kBtTmemCols = 512;
constexpr int kBtOCol = 256;
constexpr float kBtLazy = 8.0f;                      // the running maximum moves for scores this much (in log2) above it
static_assert(kBtRows == kBtKeys, "query and key tiles share a plane's size");
static_assert(16 * 8192 <= kBtStages * kBtSlot, "the softmax warps' finished rows leave through the ring");

template <bool LISTED>
__global__ void __launch_bounds__(kBtThreads, 1)
    band_attend_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                          const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_f32,
                          const __grid_constant__ CUtensorMap map_bf16, BandTcParams p) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  // full / empty: a ring slot has landed / may be overwritten; s_ready: S of a tile is there (and every product issued
  // before it is over); p_ready: P of a tile is, and O scaled; pv_done: P V of a tile is over,
  // o_done: the last one of it; q_full, drained once.
  enum { kFull = 0, kEmpty = kBtStages, kSReady = 2 * kBtStages, kPReady = kSReady + 2, kODone = kPReady + 2,
         kPvDone = kODone + 2, kQFull = kPvDone + 2, kDrained = kQFull + 1, kBars = kDrained + 1 };
  __shared__ __align__(8) uint64_t bars[kBars];
  __shared__ uint32_t tmem_base_s;
  __shared__ volatile int abort_s;
  __shared__ float swap_s[2][kBtTiles][2][kBtRows];  // by the step's parity: the maxima of a row's two threads, then their sums
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t ring = base + kBtTiles * 2 * kBtPlane;
  auto bar = [&](int i) { return smem_u32(&bars[i]); };

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // the last rows first: they see the most keys of a causal read, and the launch ends with short CTAs
  const unsigned from_last = blockIdx.x / (unsigned)p.Hq;
  const int row0 = (int)(gridDim.x / (unsigned)p.Hq - 1 - from_last) * (kBtTiles * kBtRows);  // (the caller: positions fit)
  const int head = (int)(blockIdx.x - from_last * (unsigned)p.Hq), kv_head = head / p.group;
  const int pos0 = p.first_position + row0, end_pos = p.first_position + p.R;
  const int pos_last = min(pos0 + kBtTiles * kBtRows, end_pos) - 1;
  const int band_first = LISTED ? 0 : max(0, pos0 + 1 - p.window) / kBtKeys * kBtKeys;
  const int band_tiles = (pos_last - band_first) / kBtKeys + 1;
  const bool has_sinks = !LISTED && p.sink > 0 && band_first > 0;
  const int tiles = band_tiles + (has_sinks ? 1 : 0);  // tile 0 is the sinks when there are any
  auto key0_of = [&](int n) { return has_sinks ? (n == 0 ? 0 : band_first + (n - 1) * kBtKeys) : band_first + n * kBtKeys; };
  // The last key tile that the rows of tile t walk (-1: no rows), and whether they walk tile n: the sinks, and from the
  // first row's window to the last row.
  auto last_of = [&](int t) {
    const int first = pos0 + t * kBtRows, last = min(first + kBtRows, end_pos) - 1;
    return first >= end_pos ? -1 : (last - band_first) / kBtKeys + (has_sinks ? 1 : 0);
  };
  const int lasts[kBtTiles] = {last_of(0), last_of(1)};
  auto sees = [&](int t, int n) {
    const int last = t == 0 ? lasts[0] : lasts[1];
    if (n >= last) return n == last;
    // (where the first key tile is the band's own, it holds the sinks as well)
    return LISTED || (n == 0 && p.sink > 0 && key0_of(0) == 0) || key0_of(n) + kBtKeys > pos0 + t * kBtRows + 1 - p.window;
  };

  if (threadIdx.x == 0) {
    for (int i = 0; i < kBars; ++i) mbar_init(bar(i), i >= kPReady && i < kODone ? 2 * kBtRows : 1);
    abort_s = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)),
                 "r"(kBtTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = tmem_base_s;

  if (warp < 2) {
    if (warp == 0 && lane == 0) {
      mbar_expect_tx(bar(kQFull), kBtTiles * 2 * kBtPlane);  // (rows past the last are filled with zeros)
#pragma unroll
      for (int t = 0; t < kBtTiles; ++t)
#pragma unroll
        for (int plane = 0; plane < 2; ++plane)
          tma_load_2d(base + (2 * t + plane) * kBtPlane, &map_q, bar(kQFull), head * 128 + 64 * plane, row0 + t * kBtRows);
      int sent = 0;
      bool ok = true;
      auto send = [&](const CUtensorMap *map, int n) {
        const int slot = sent % kBtStages;
        if (sent >= kBtStages) ok = !abort_s && mbar_wait(bar(kEmpty + slot), (sent / kBtStages + 1) & 1);
        if (!ok) return;
        const uint32_t dst = ring + slot * kBtSlot;
        const int y = key0_of(n), x = kv_head * 128;
        mbar_expect_tx(bar(kFull + slot), kBtSlot);
        tma_load_2d(dst, map, bar(kFull + slot), x, y);
        tma_load_2d(dst + kBtPlane, map, bar(kFull + slot), x + 64, y);
        ++sent;
      };
      for (int n = 0; n <= tiles && ok; ++n) {  // K 0, K 1, V 0, K 2, V 1, ...: what a step of the issuing warp needs
        if (n < tiles) send(&map_k, n);
        if (n > 0 && ok) send(&map_v, n - 1);
      }
      if (!ok) abort_s = 1;
      // nothing of this CTA's copies may be under way when it leaves: the last one of every slot has landed
      mbar_wait(bar(kQFull), 0);
      for (int i = max(0, sent - kBtStages); i < sent; ++i) mbar_wait(bar(kFull + i % kBtStages), (i / kBtStages) & 1);
    } else if (warp == 1) {
      // (What this warp does between two tiles' products is time the tensor pipe waits: it shares its scheduler with four
      // warps of softmax and gets an instruction in some twenty cycles. So slots, phases and descriptors are kept, not
      // computed, and the abort flag is looked at only by a wait that waits.)
      const uint32_t idesc_s = umma_idesc(kBtKeys), idesc_o = umma_idesc(128, true);
      const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_base, 0), bars_at = bar(0);
      const uint64_t q_desc = smem_desc_sw128(base), k_desc = smem_desc_sw128(ring), v_desc = smem_desc_mn_sw128(ring, kBtPlane);
      constexpr uint32_t kSlotUnits = kBtSlot >> 4;
      auto wait = [&](int i, uint32_t parity) { return mbar_wait_warp(bars_at + 8 * i, parity, &abort_s); };
      bool ok = wait(kQFull, 0);
      uint32_t slot = 0, ring_phase = 0;          // the next ring slot and its parity
      uint32_t p_phase = 0;                       // bit t: parity of tile t's P
      bool started[kBtTiles] = {false, false};    // whether O of a tile holds anything
      uint32_t pending = 0;                       // bit t: tile t's P V of the key tile before is to come
      for (int n = 0; n <= tiles && ok; ++n) {
        uint32_t k_at = 0, v_at = 0;
        if (n < tiles) {
          ok = wait(kFull + slot, ring_phase);
          k_at = slot;
          if (++slot == kBtStages) slot = 0, ring_phase ^= 1;
        }
        if (n > 0 && ok) {
          ok = wait(kFull + slot, ring_phase);
          v_at = slot;
          if (++slot == kBtStages) slot = 0, ring_phase ^= 1;
        }
        if (!ok) break;
        const uint64_t k_tile = k_desc + k_at * kSlotUnits, v_tile = v_desc + v_at * kSlotUnits;
        const uint32_t seen = (sees(0, n) ? 1u : 0u) | (sees(1, n) ? 2u : 0u);
#pragma unroll
        for (int t = 0; t < kBtTiles; ++t) {
          const uint32_t s_col = tmem + t * kBtKeys, o_col = tmem + kBtOCol + t * 128;
          if (pending >> t & 1) {
            ok = ok && wait(kPReady + t, p_phase >> t & 1);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (elect_one()) {
#pragma unroll
              for (int half = 0; half < 2; ++half)
#pragma unroll
                for (int term = 0; term < 2; ++term)
#pragma unroll
                  for (int k = 0; k < 4; ++k)  // 16 keys: 8 columns of P, 2,048 bytes down a plane of V
                    umma_bf16_ts(o_col, s_col + 64 * half + 32 * (k >> 1) + 16 * term + 8 * (k & 1),
                                 v_tile + (4 * half + k) * (2048 >> 4), idesc_o, (half | term | k) != 0 || started[t]);
              umma_commit(bars_at + 8 * ((n > lasts[t] ? kODone : kPvDone) + t));
            }
            __syncwarp();
            // S of the next keys is written over the P that these products read: they have to be over. (Products are kept in
            // order by themselves only where they have one accumulator and one shape.)
            if (n <= lasts[t]) ok = wait(kPvDone + t, p_phase >> t & 1);
            p_phase ^= 1u << t, started[t] = true;
          }
          if (ok && n < tiles && (seen >> t & 1)) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (elect_one()) {
#pragma unroll
              for (int plane = 0; plane < 2; ++plane)
#pragma unroll
                for (int k = 0; k < 4; ++k)
                  umma_bf16(s_col, q_desc + ((2 * t + plane) * kBtPlane >> 4) + 2 * k, k_tile + (plane * kBtPlane >> 4) + 2 * k,
                            idesc_s, (plane | k) != 0);
              umma_commit(bars_at + 8 * (kSReady + t));
            }
            __syncwarp();
          }
        }
        pending = n < tiles ? seen : 0;
        if (elect_one()) {
          if (n < tiles) umma_commit(bars_at + 8 * (kEmpty + k_at));
          if (n > 0) umma_commit(bars_at + 8 * (kEmpty + v_at));
        }
        __syncwarp();
      }
      if (!ok) {  // every product of this CTA's is over before its tensor memory goes
        abort_s = 1;
        if (elect_one()) umma_commit(bar(kDrained));
        mbar_wait(bar(kDrained), 0);
      }
    }
  } else {
    const int t = (warp - 2) >> 3, half = ((warp - 2) >> 2) & 1, quarter = warp & 3;  // (a warp reaches its quarter of the lanes)
    const int row = quarter * 32 + lane;
    const uint32_t lane_addr = tmem_base + ((uint32_t)(quarter * 32) << 16);
    const uint32_t s_col = lane_addr + t * kBtKeys + half * 64, o_col = lane_addr + kBtOCol + t * 128 + half * 64;
    auto pair_sync = [&] { asm volatile("bar.sync %0, 64;" ::"r"(1 + t * 4 + quarter) : "memory"); };  // the two warps of 32 rows
    const int tile_pos0 = pos0 + t * kBtRows, pos = tile_pos0 + row, in_call = row0 + t * kBtRows + row;
    const int tile_last = min(tile_pos0 + kBtRows, end_pos) - 1;
    const bool live = in_call < p.R;
    const int start = max(0, pos + 1 - p.window);
    // a tile inside every row's window, below every row's position and inside the cache needs no masks
    const int inside_from = max(0, tile_last + 1 - p.window);
    const uint64_t scale2 = pair_of(p.scale_log2, p.scale_log2), minus_one2 = pair_of(-1.0f, -1.0f);
    float m_ref = -INFINITY;  // the point the exponents are taken from, in log2
    uint64_t l2[2] = {0, 0};  // the row's sum, four of it side by side
    int steps = 0;
    bool go = true;
    for (int n = 0; n < tiles; ++n) {
      if (!sees(t, n)) continue;
      const int key0 = key0_of(n);
      uint32_t words[2] = {0u, 0u};  // a bit a key of this thread's 64: whether the row reads it
      bool masked = true;
      if constexpr (LISTED) {
        if (live) {
          const uint2 w = reinterpret_cast<const uint2 *>(p.mask + (int64_t)n * p.R + in_call)[half];
          words[0] = w.x, words[1] = w.y;
        }
        masked = !__all_sync(0xffffffffu, (words[0] & words[1]) == 0xffffffffu);
      } else {
        const bool is_sinks = has_sinks && n == 0;
        masked = is_sinks || key0 < inside_from || key0 + kBtKeys - 1 > tile_pos0 || key0 + kBtKeys > p.n_keys;
        if (masked) {
          const int first = key0 + half * 64;
          auto rel = [&](int key) { return max(-1, min(64, key - first)); };
          const int end = live ? rel(p.n_keys) : 0;                   // columns at or past it are outside the cache
          const int sinks = rel(min(p.sink, start));                   // columns below it are the row's sinks
          const int from = is_sinks ? 64 : rel(start), to = is_sinks ? -1 : rel(pos);  // the window: from <= c <= to
          auto below = [](int x) { return x >= 32 ? 0xffffffffu : (x <= 0 ? 0u : (1u << x) - 1u); };
#pragma unroll
          for (int c = 0; c < 2; ++c)
            words[c] = ((below(to + 1 - 32 * c) & ~below(from - 32 * c)) | below(sinks - 32 * c)) & below(end - 32 * c);
        }
      }
      go = go && __all_sync(0xffffffffu, !abort_s && mbar_wait(bar(kSReady + t), steps & 1));
      if (!go) {  // (a warp that gave up walks on: it owes the row's other threads a barrier a step)
        pair_sync();
        ++steps;
        continue;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      // keys 32 c .. 32 c + 31 of this thread's, the masked ones at -inf (taken twice, for the maximum and for the
      // exponentials: 64 scores held in between are more registers than eighteen warps leave a thread)
      auto load_keys = [&](int c, uint32_t (&sv)[32]) {
        tmem_load_32(s_col + 32 * c, sv);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (masked) {
          const uint32_t w = words[c];
#pragma unroll
          for (int i = 0; i < 32; ++i) sv[i] = (w & (1u << i)) ? sv[i] : 0xff800000u;  // -inf
        }
      };
      float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t sv[32];
        load_keys(c, sv);
#pragma unroll
        for (int i = 0; i < 32; i += 2)
          m4[(i >> 1) & 3] = fmaxf(fmaxf(m4[(i >> 1) & 3], __uint_as_float(sv[i])), __uint_as_float(sv[i + 1]));
      }
      float m_tile = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3]));
      swap_s[steps & 1][t][half][row] = m_tile;
      pair_sync();
      m_tile = fmaxf(m_tile, swap_s[steps & 1][t][half ^ 1][row]) * p.scale_log2;  // (the scale is positive)
      if (__any_sync(0xffffffffu, m_tile > m_ref + kBtLazy)) {
        const float m_new = fmaxf(m_ref, m_tile);
        const float alpha = m_new == m_ref ? 1.0f : fast_exp2(m_ref - m_new);
        m_ref = m_new;
        const uint64_t alpha2 = pair_of(alpha, alpha), zero2 = pair_of(0.0f, 0.0f);
        l2[0] = fma_pair(l2[0], alpha2, zero2), l2[1] = fma_pair(l2[1], alpha2, zero2);
        if (steps > 0) {
#pragma unroll 1
          for (int c = 0; c < 64; c += 32) {
            uint32_t o[32];
            tmem_load_32(o_col + c, o);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
            tmem_store_32(o_col + c, o);
          }
        }
      }
      const float off = m_ref == -INFINITY ? 0.0f : -m_ref;
      const uint64_t off2 = pair_of(off, off);
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t sv[32], hi[16], lo[16];
        load_keys(c, sv);
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          float e0, e1;
          split_pair(fma_pair(pair_of(__uint_as_float(sv[2 * i]), __uint_as_float(sv[2 * i + 1])), scale2, off2), e0, e1);
          e0 = fast_exp2(e0), e1 = fast_exp2(e1);
          const uint64_t e2 = pair_of(e0, e1);
          l2[i & 1] = add_pair(l2[i & 1], e2);
          hi[i] = pack_bf16x2(e0, e1);
          float r0, r1;
          split_pair(fma_pair(pair_of(__uint_as_float(hi[i] << 16), __uint_as_float(hi[i] & 0xffff0000u)), minus_one2, e2),
                     r0, r1);
          lo[i] = pack_bf16x2(r0, r1);
        }
        tmem_store_16(s_col + 32 * c, hi);
        tmem_store_16(s_col + 32 * c + 16, lo);
      }
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar(kPReady + t)) : "memory");
      ++steps;
    }
    float a, b, c, d;
    split_pair(l2[0], a, b);
    split_pair(l2[1], c, d);
    float l_row = (a + b) + (c + d);
    swap_s[steps & 1][t][half][row] = l_row;
    pair_sync();
    l_row += swap_s[steps & 1][t][half ^ 1][row];
    // (both tiles' last products: the ring is written over below)
    for (int i = 0; i < kBtTiles; ++i)
      if (go && lasts[i] >= 0) go = __all_sync(0xffffffffu, !abort_s && mbar_wait(bar(kODone + i), 0));
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (go) {
      const float inv = l_row > 0.0f ? 1.0f / l_row : 0.0f;
      const int64_t out_row = (int64_t)in_call * p.Hq + head;
      bool finite = true;
      // The rows leave through shared memory, a box of 32 rows by 128 bytes a copy: a warp's stores of its own rows touched 32
      // lines each and were 21 of a band CTA's 75 k cycles. (Key and value tiles are spent when both tiles' last products
      // are over; boxes are cut at the last row of the call.)
      const uint32_t box = ring + (warp - 2) * 8192;
      auto row_at = [&](int piece) { return box + (piece >> 3) * 4096 + lane * 128 + (((piece & 7) ^ (lane & 7)) << 4); };
      const int x0 = head * 128 + half * 64, y0 = row0 + t * kBtRows + quarter * 32;
      float x[2][32];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        uint32_t r[32];
        if (steps > 0) {
          tmem_load_32(o_col + 32 * e, r);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        }
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          x[e][i] = steps > 0 ? __uint_as_float(r[i]) * inv : 0.0f;
          finite = finite && isfinite(x[e][i]);
        }
      }
      auto store = [&](uint32_t at, uint32_t w0, uint32_t w1, uint32_t w2, uint32_t w3) {
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(w0), "r"(w1), "r"(w2), "r"(w3) : "memory");
      };
      if (p.out) {
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const float *f = &x[i >> 3][(i & 7) * 4];
          store(row_at(i), __float_as_uint(f[0]), __float_as_uint(f[1]), __float_as_uint(f[2]), __float_as_uint(f[3]));
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane < 2 && y0 < p.R) {
          tma_store_2d(&map_f32, box + lane * 4096, x0 + lane * 32, y0);
          tma_store_read();
        }
        __syncwarp();
      }
      if (p.out_bf16) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float *f = &x[i >> 2][(i & 3) * 8];
          store(row_at(i), pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]), pack_bf16x2(f[4], f[5]), pack_bf16x2(f[6], f[7]));
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0 && y0 < p.R) {
          tma_store_2d(&map_bf16, box, x0, y0);
          tma_store_read();
        }
        __syncwarp();
      }
      if (live && half == 0 && p.lse)
        p.lse[out_row] = l_row > 0.0f ? (m_ref + log2f(l_row)) * 0.6931471805599453f : -INFINITY;
      if (live && p.not_finite && !(finite && isfinite(l_row))) *p.not_finite = 1;
    } else {
      abort_s = 1;
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kBtTmemCols));
  }
  if (threadIdx.x == 0 && abort_s && p.status) atomicAdd(p.status, 1);
}

int launch_band_attend_tc(const BandTcCall &c, cudaStream_t stream) {
  CUtensorMap map_q, map_k, map_v, map_f32 = {}, map_bf16 = {};
  const int64_t width = (int64_t)c.p.Hq * 128;
  int rc = make_map(&map_q, c.q, c.p.R, width, c.q_row_stride, kBtRows);
  if (rc == LSA_OK) rc = make_map(&map_k, c.k, c.p.n_keys, (int64_t)c.Hkv * 128, c.kv_row_stride, kBtKeys);
  if (rc == LSA_OK) rc = make_map(&map_v, c.v, c.p.n_keys, (int64_t)c.Hkv * 128, c.kv_row_stride, kBtKeys);
  // (the outputs, in boxes of a warp's rows)
  if (rc == LSA_OK && c.p.out) rc = make_map_of(&map_f32, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, c.p.out, c.p.R, width, width, 32);
  if (rc == LSA_OK && c.p.out_bf16) rc = make_map(&map_bf16, c.p.out_bf16, c.p.R, width, width, 32);
  if (rc != LSA_OK) return rc;
  auto kernel = c.p.mask ? band_attend_tc_kernel<true> : band_attend_tc_kernel<false>;
  if (!allow_shared(kernel, kBtSmem)) return LSA_ERR_LAUNCH;
  const int64_t blocks = ((int64_t)c.p.R + kBtTiles * kBtRows - 1) / (kBtTiles * kBtRows);
  if (blocks * c.p.Hq > INT32_MAX) return LSA_ERR_ARGUMENT;
  kernel<<<(unsigned)(blocks * c.p.Hq), kBtThreads, kBtSmem, stream>>>(map_q, map_k, map_v, map_f32, map_bf16, c.p);
  LSA_LAUNCH_CHECK();
  return LSA_OK;
}

}  // namespace lsa
