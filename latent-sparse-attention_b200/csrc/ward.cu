// Capped Ward bucketing of cluster blocks of up to 4,096 pools with 16, 32 or 64 index dims: the buckets of a cache,
// and the node-bucket pairings of the tree over them.
//
// A block of up to 512 pools is merged from its first round to its last by a cluster of 1 to 8 CTAs, a larger one by a cluster
// or by up to as many CTAs as there are SMs. Every CTA keeps the block's per-row state (sizes, norms, cheapest partner, who is
// alive) in its own shared memory and takes every decision itself, so only two things cross between the CTAs of a round: the
// cheapest partners (64-bit minima, the greater word the cost and the lower the partner, so that a tie goes to the lower row
// whatever the order of arrival) and the merged rows. In the smaller blocks every CTA keeps the minima of the pairs it looked
// at, reads the others' through distributed shared memory and merges every row itself; in the larger ones the key sums do not
// fit beside the rest, and both live in the workspace.
//
// A round looks only at what the round before changed. A pair's cost depends on nothing but its two rows, so a row whose
// cheapest partner neither merged nor went keeps it, unless a row that just merged is cheaper:
//   dirty rows (merged, or their partner merged or went)  x  all open rows
// and a row too large for the smallest row left is closed: it can never merge again (in a pairing, every pair). A pair's
// cost has the same bits from either side, so two dirty rows meet once and a tile of theirs serves both, and the other open
// rows learn of what merged from the same tiles. What bounds the first rounds is a warp's way through a tile (of a
// larger block's tile of 128 x 128 pairs, 23 k cycles, the products are 13.5 k, where their multiply-adds alone would be 8 k,
// and the costs 5 k; two sums a multiply-add with fma.rn.f32x2, lanes that share operands so that these leave shared memory in
// three quarters of the time, and two teams of warps with a tile each came out alike or slower), the last ones barriers, where a handful of rows is dirty (a round of a block of 80 pools takes 7 us, of which the tiles are 2).
// Measured on a B200, against every row searching all of its partners every round (one CTA a block up to 512 pools, two
// launches a round, 256 rounds, above): the pairings of 16 blocks of 4,096, 2,048 and 1,024 buckets 26.0 -> 4.4 ms; 1,024
// blocks of 256 pools with the pairings of 512, 256 and 128 buckets 7.2 -> 2.4 ms; 9 blocks of 128 pools 165 -> 57 us; one
// block of 80 pools, sixteen rounds, 190 -> 119 us. With every pair once, on the index of 1M clustered tokens: 1,024 blocks of 256
// pools 2.10 -> 1.65 ms, the pairings of 16 blocks of 4,096 buckets 3.07 -> 2.28 (the first round 1.30 -> 0.76), of 2,048 0.92 ->
// 0.77, of 1,024 384 -> 353 us, of 512 176 -> 158. With the dirty and the steady partners as one run of tiles, a last row tile's few
// rows over all warps, and one branch for a lane's pairs of a row, 1,024 blocks of 256 pools 1.66 -> 1.47 ms, the pairings of 4,096
// buckets 2.28 -> 2.21, of 1,024 352 -> 335 us.
//
// Arithmetic order is the CPU specification's: a dot is an fma chain in ascending dim order, costs are evaluated as
// written, so labels are bit-equal to a replay in that order.
#include <cooperative_groups.h>

#include <type_traits>

#include "common.cuh"

namespace lsa {

namespace cg = cooperative_groups;

// A tile: eight rows a warp (two where the warps have no more to share), and as many partners as the eight of all warps (a
// lane takes every 32nd).
constexpr int kWardRows = 8, kWardFewRows = 2;
__host__ __device__ constexpr int ward_threads(bool local) { return local ? 256 : 512; }
__host__ __device__ constexpr int ward_tile(bool local) { return kWardRows * ward_threads(local) / 32; }
constexpr int kWardMaxCtas = 8;      // a cluster's portable size
constexpr int kWardMaxPools = 4096;  // pools of a block, at most
constexpr int kWardApart = 64;       // ints from one block's counter of arrivals to the next (nothing else in its cache lines)
constexpr int kWardPatience = 1 << 24;  // looks at the counter before a wait gives up (seconds)
constexpr int kWardLocalPools = 512;  // blocks up to this many pools keep their key sums in every CTA's shared memory

enum : uint8_t { kAlive = 1, kOpen = 2, kChanged = 4, kMerged = 8 };

struct WardParams {
  const float *pool_keys;   // [G, P, D]
  const float *pool_sizes;  // [G, P] or NULL
  float uniform_size, bucket_cap;
  int P, bucket_count, max_rounds;
  int64_t *labels;    // [G, P]
  uint8_t *reached;   // [G]
  int32_t *rounds;    // [G] or NULL
  // the workspace of larger blocks: key sums [G, P, D], squared norms and norms [G, P], cheapest partners [2, G, P], and where
  // a block's CTAs are no cluster how many of them arrived at its barriers [G, kWardApart] (zero at launch; else NULL)
  float *sums, *sq, *al;
  unsigned long long *cheapest;
  int *arrived;
  int ctas;  // CTAs a block
};

// A CTA's shared memory, carved from the dynamic part.
template <int D, bool LOCAL>
struct WardShared {
  static constexpr int TILE = ward_tile(LOCAL);
  static constexpr int LD = D + 4;  // keeps float4 alignment and spreads consecutive rows over the banks
  unsigned long long *cheapest;  // [1 or 2][P] (cost, partner) a row, of the pairs this CTA looked at
  float *a, *b;                     // [tile][LD]
  float *sums;                      // [P][LD] of a local block
  float *sz, *sq, *al, *cost;       // [P]
  uint16_t *best, *parent;          // [P]
  uint16_t *dirty, *steady, *merged, *pairs;  // [P] lists of rows
  uint8_t *flag;                    // [P]

  // (bytes, and with `base` the pointers)
  __host__ __device__ size_t carve(unsigned char *base, int P, bool two) {
    size_t at = 0;
    auto take = [&](size_t bytes) {
      unsigned char *p = base + at;
      at += (bytes + 15) & ~(size_t)15;
      return p;
    };
    cheapest = LOCAL ? (unsigned long long *)take((size_t)P * 8 * (two ? 2 : 1)) : nullptr;
    a = (float *)take(sizeof(float) * TILE * LD);
    b = (float *)take(sizeof(float) * TILE * LD);
    sums = LOCAL ? (float *)take(sizeof(float) * P * LD) : nullptr;
    sz = (float *)take((size_t)P * 4), sq = (float *)take((size_t)P * 4);
    al = (float *)take((size_t)P * 4), cost = (float *)take((size_t)P * 4);
    best = (uint16_t *)take((size_t)P * 2), parent = (uint16_t *)take((size_t)P * 2);
    dirty = (uint16_t *)take((size_t)P * 2), steady = (uint16_t *)take((size_t)P * 2);
    merged = (uint16_t *)take((size_t)P * 2), pairs = (uint16_t *)take((size_t)P * 2);
    flag = (uint8_t *)take((size_t)P);
    return at;
  }
};

// A (cost, partner) as one number of the same order. (-0 and 0 are one cost: adding 0 makes them one number.)
__device__ __forceinline__ unsigned long long pack_cheapest(float cost, int partner) {
  return ((unsigned long long)((uint32_t)ordered_bits(__fadd_rn(cost, 0.0f)) ^ 0x80000000u) << 32) | (uint32_t)partner;
}
__device__ __forceinline__ float cheapest_cost(unsigned long long packed) {
  const int32_t bits = (int32_t)((uint32_t)(packed >> 32) ^ 0x80000000u);
  return __int_as_float(bits < 0 ? (bits ^ 0x7FFFFFFF) : bits);
}

// Squared norm of a row as one fma chain, sixteen bytes at a time.
template <int D>
__device__ __forceinline__ float row_square(const float4 *row) {
  float s = 0.0f;
#pragma unroll
  for (int k = 0; k < D / 4; ++k) {
    s = fmaf(row[k].x, row[k].x, s), s = fmaf(row[k].y, row[k].y, s);
    s = fmaf(row[k].z, row[k].z, s), s = fmaf(row[k].w, row[k].w, s);
  }
  return s;
}

template <int D, bool LOCAL>
__global__ void __launch_bounds__(ward_threads(LOCAL), LOCAL ? 2 : 1) ward_kernel(WardParams p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cg::cluster_group cluster = cg::this_cluster();
  constexpr int kThreads = ward_threads(LOCAL), TILE = ward_tile(LOCAL), LD = D + 4, COLS = TILE / 32;
  const int ctas = p.ctas, rank = (int)(blockIdx.x % ctas);
  const int64_t g = blockIdx.x / ctas;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, P = p.P;
  const unsigned below = (1u << lane) - 1;
  WardShared<D, LOCAL> s;
  s.carve(smem_raw, P, ctas > 1);
  // The minima of even and odd rounds lie apart: the others may still be reading the last round's when the next's are
  // set up.
  const int64_t apart = LOCAL ? (ctas > 1 ? P : 0) : (int64_t)(gridDim.x / ctas) * P;
  unsigned long long *mine = LOCAL ? s.cheapest : p.cheapest + g * P;
  __shared__ int warp_count[kThreads / 32], n_merge_s, smallest_s;
  __shared__ float bound_s[TILE], known_s[TILE];  // costs that the cheapest of a tile's rows and of its partners are not above
  // What a CTA wrote before is seen by all of the block's after. (CTAs that are no cluster are launched as a cooperative grid,
  // so that all of them run: a wait that gives up all the same ends the block as one that did not reach its count.)
  bool gave_up = false;
  int due = 0;
  auto everyone = [&] {
    if (ctas == 1) {
      __syncthreads();
    } else if (LOCAL || !p.arrived) {
      cluster.sync();
    } else {
      __syncthreads();
      due += ctas;
      int late = 0;
      if (tid == 0) {
        volatile int *arrived = p.arrived + g * kWardApart;
        __threadfence();
        atomicAdd((int *)arrived, 1);
        late = 1;
        for (int look = 0; late && look < kWardPatience; ++look) late = *arrived < due;
        __threadfence();
      }
      gave_up = __syncthreads_or(late);
    }
  };
  const float *src = p.pool_keys + g * (int64_t)P * D;
  float *sums_g = LOCAL ? nullptr : p.sums + g * (int64_t)P * D;
  float *sq_g = LOCAL ? nullptr : p.sq + g * P, *al_g = LOCAL ? nullptr : p.al + g * P;

  // ---- the block as it starts
  if (tid == 0) smallest_s = 0x7FFFFFFF;
  if (LOCAL) {
    for (int e = tid; e < P * (D / 4); e += kThreads) {
      const int i = e / (D / 4), k = e - i * (D / 4);
      *reinterpret_cast<float4 *>(s.sums + (size_t)i * LD + 4 * k) = *reinterpret_cast<const float4 *>(src + (size_t)i * D + 4 * k);
    }
    __syncthreads();
    for (int i = tid; i < P; i += kThreads) {
      float4 row[D / 4];
#pragma unroll
      for (int k = 0; k < D / 4; ++k) row[k] = *reinterpret_cast<const float4 *>(s.sums + (size_t)i * LD + 4 * k);
      const float q = row_square<D>(row);
      s.sq[i] = q, s.al[i] = sqrtf(q > 0.0f ? q : 0.0f);
    }
  } else {
    for (int i = rank * kThreads + tid; i < P; i += ctas * kThreads) {
      float4 row[D / 4];
#pragma unroll
      for (int k = 0; k < D / 4; ++k) {
        row[k] = *reinterpret_cast<const float4 *>(src + (size_t)i * D + 4 * k);
        *reinterpret_cast<float4 *>(sums_g + (size_t)i * D + 4 * k) = row[k];
      }
      const float q = row_square<D>(row);
      sq_g[i] = q, al_g[i] = sqrtf(q > 0.0f ? q : 0.0f);
    }
  }
  for (int i = tid; i < P; i += kThreads) {
    s.sz[i] = p.pool_sizes ? p.pool_sizes[g * P + i] : p.uniform_size;
    s.parent[i] = (uint16_t)i;
    s.flag[i] = kAlive | kChanged;
  }
  __syncthreads();

  int n_alive = P, rounds = 0, n_dirty = 0, n_steady = 0, n_merged = 0, side = 0;
  // The lists of the coming round, ascending: which rows are open (a row and the smallest row fit under the cap), and
  // of them the dirty, the steady and the just merged. Every CTA makes the same lists.
  auto make_lists = [&] {
    int32_t least = 0x7FFFFFFF;
    for (int i = tid; i < P; i += kThreads)
      if (s.flag[i] & kAlive) least = min(least, ordered_bits(isnan(s.sz[i]) ? -INFINITY : s.sz[i]));
    least = __reduce_min_sync(0xffffffffu, least);
    if (lane == 0) atomicMin(&smallest_s, least);
    __syncthreads();
    const int32_t bits = smallest_s;
    float smallest = __int_as_float(bits < 0 ? (bits ^ 0x7FFFFFFF) : bits);
    if (smallest < 0.0f) smallest = -INFINITY;  // (a size may shrink then: nothing is closed for good)
    n_dirty = n_steady = n_merged = 0;
    for (int i0 = 0; i0 < P; i0 += kThreads) {
      const int i = i0 + tid;
      bool is_dirty = false, is_steady = false, is_merged = false;
      if (i < P) {
        const uint8_t f = s.flag[i];
        const bool open = (f & kAlive) && !(__fadd_rn(s.sz[i], smallest) > p.bucket_cap);
        if (open) {
          is_dirty = (f & kChanged) || (s.cost[i] < INFINITY && (s.flag[s.best[i]] & kChanged));
          is_steady = !is_dirty;
          is_merged = f & kMerged;
        }
      }
      static_assert(kThreads < 1024, "three sums of up to kThreads in a word");
      const unsigned vd = __ballot_sync(0xffffffffu, is_dirty), vs = __ballot_sync(0xffffffffu, is_steady);
      const unsigned vm = __ballot_sync(0xffffffffu, is_merged);
      if (lane == 0) warp_count[warp] = __popc(vd) | __popc(vs) << 10 | __popc(vm) << 20;  // (ten bits a sum: the threads of the CTA at most)
      __syncthreads();
      int before = 0, all = 0;
#pragma unroll
      for (int w = 0; w < kThreads / 32; ++w) {
        if (w < warp) before += warp_count[w];
        all += warp_count[w];
      }
      if (is_dirty) s.dirty[n_dirty + (before & 1023) + __popc(vd & below)] = (uint16_t)i;
      if (is_steady) s.steady[n_steady + (before >> 10 & 1023) + __popc(vs & below)] = (uint16_t)i;
      if (is_merged) s.merged[n_merged + (before >> 20) + __popc(vm & below)] = (uint16_t)i;
      n_dirty += all & 1023, n_steady += all >> 10 & 1023, n_merged += all >> 20;
      __syncthreads();
    }
    // What the flags say of the last round is used up; who is open is written for the read of the minima. (A row's
    // next minimum: none yet for a dirty row, what it has for a steady one.)
    for (int i = tid; i < P; i += kThreads) s.flag[i] &= kAlive;
    __syncthreads();
    for (int e = tid; e < n_dirty; e += kThreads) {
      const int i = s.dirty[e];
      s.flag[i] |= kOpen;
      if (LOCAL || e % ctas == rank) mine[side * apart + i] = ~0ull;
    }
    for (int e = tid; e < n_steady; e += kThreads) {
      const int i = s.steady[e];
      s.flag[i] |= kOpen;
      if (LOCAL || e % ctas == rank) mine[side * apart + i] = s.cost[i] < INFINITY ? pack_cheapest(s.cost[i], s.best[i]) : ~0ull;
    }
    if (tid == 0) smallest_s = 0x7FFFFFFF;
  };

  for (int i = tid; i < P; i += kThreads) s.cost[i] = INFINITY, s.best[i] = 0;
  __syncthreads();
  make_lists();
  everyone();
  if (!LOCAL) {
    for (int i = tid; i < P; i += kThreads) s.sq[i] = __ldcg(sq_g + i), s.al[i] = __ldcg(al_g + i);
    __syncthreads();
  }

  // A merged row's norm is at most the block's norms together: 4,096 of up to 1e15 keep `both` under 1e19, whose square is in
  // range. (Norms that are not numbers count as greater; an infinite slack leaves `most` infinitely below zero, or no number.)
  bool great = false;
  for (int i = tid; i < P; i += kThreads) great = great || !(s.al[i] <= 1e15f);
  const float keep = __syncthreads_or(great) ? -INFINITY : 1.0f - 9.5367431640625e-7f;

  for (; rounds < p.max_rounds && n_alive > p.bucket_count && !gave_up; ++rounds) {
    // ---- the cheapest partners: tiles of (dirty x open), dealt to the CTAs in runs. A pair's cost is the same from either side,
    // bit for bit, so a tile serves its rows and its partners: two dirty rows meet once, and a steady row meets what merged.
    const int n_open = n_dirty + n_steady;
    auto open_row = [&](int at) { return at < n_dirty ? s.dirty[at] : s.steady[at - n_dirty]; };  // (no tile ends with the dirty ones)
    auto stage = [&](float *tile, int from, int n, int most) {
      for (int e = tid; e < most * (D / 4); e += kThreads) {
        const int r = e / (D / 4), k = e - r * (D / 4);
        if (from + r < n) {
          const int id = open_row(from + r);
          *reinterpret_cast<float4 *>(tile + r * LD + 4 * k) =
              LOCAL ? *reinterpret_cast<const float4 *>(s.sums + (size_t)id * LD + 4 * k)
                    : __ldcg(reinterpret_cast<const float4 *>(sums_g + (size_t)id * D + 4 * k));
        }
      }
    };
    // A cost that a row's cheapest is not above: what it has so far.
    auto known = [&](int id) {
      const unsigned long long *at = mine + side * apart + id, v = LOCAL ? *(const volatile unsigned long long *)at : __ldcg(at);
      return v == ~0ull ? INFINITY : cheapest_cost(v);
    };
    // One row tile of the dirty rows against partner tiles first_tile .. end_tile - 1 of the dirty and then the steady rows.
    auto search = [&](auto rows_a_warp, int first_row, int first_tile, int end_tile) {
      constexpr int ROWS = decltype(rows_a_warp)::value;
      const uint16_t *my_list = s.dirty + first_row + warp * ROWS;
      const int my_rows = min(ROWS, n_dirty - first_row - warp * ROWS);  // (0 or less: this warp has none)
      float best_c[ROWS];
      int best_j[ROWS];
#pragma unroll
      for (int i = 0; i < ROWS; ++i) best_c[i] = INFINITY, best_j[i] = 0x7FFFFFFF;
      __syncthreads();  // (the tiles are free)
      stage(s.a, first_row, n_dirty, ROWS * kThreads / 32);
      if (lane < my_rows) bound_s[warp * ROWS + lane] = known(my_list[lane]);
      for (int t = first_tile; t < end_tile; ++t) {
        const int from = t * TILE;
        // (the dirty rows of the tile that the rows are of meet themselves: every pair is there twice)
        const int one_way = t == first_row / TILE ? n_dirty : 0;
        if (t > first_tile) __syncthreads();
        stage(s.b, from, n_open, TILE);
        if (tid < TILE) known_s[tid] = from + tid >= one_way && from + tid < n_open ? known(open_row(from + tid)) : -INFINITY;
        __syncthreads();
        if (my_rows <= 0) continue;
        float acc[ROWS][COLS];
#pragma unroll
        for (int i = 0; i < ROWS; ++i)
#pragma unroll
          for (int j = 0; j < COLS; ++j) acc[i][j] = 0.0f;
#pragma unroll 4
        for (int k = 0; k < D; k += 4) {
          float4 b[COLS];
#pragma unroll
          for (int j = 0; j < COLS; ++j) b[j] = *reinterpret_cast<const float4 *>(s.b + (lane + 32 * j) * LD + k);
#pragma unroll
          for (int i = 0; i < ROWS; ++i) {
            const float4 a = *reinterpret_cast<const float4 *>(s.a + (warp * ROWS + i) * LD + k);
#pragma unroll
            for (int j = 0; j < COLS; ++j) {
              acc[i][j] = fmaf(a.x, b[j].x, acc[i][j]);
              acc[i][j] = fmaf(a.y, b[j].y, acc[i][j]);
              acc[i][j] = fmaf(a.z, b[j].z, acc[i][j]);
              acc[i][j] = fmaf(a.w, b[j].w, acc[i][j]);
            }
          }
        }
        // (rows and partners past the lists hold whatever the tiles held: they are not looked at)
        int id_j[COLS], theirs_i[COLS];
        float sq_j[COLS], al_j[COLS], sz_j[COLS], theirs_c[COLS];
#pragma unroll
        for (int j = 0; j < COLS; ++j) {
          const int c = from + lane + 32 * j;
          id_j[j] = c < n_open ? open_row(c) : -1;
          sq_j[j] = c < n_open ? s.sq[id_j[j]] : 0.0f;
          al_j[j] = c < n_open ? s.al[id_j[j]] : 0.0f;
          sz_j[j] = c < n_open ? s.sz[id_j[j]] : 0.0f;
          theirs_c[j] = known_s[lane + 32 * j], theirs_i[j] = -1;
        }
#pragma unroll
        for (int i = 0; i < ROWS; ++i) {
          if (i >= my_rows) break;
          const int id_i = my_list[i];
          const float sq_i = s.sq[id_i], al_i = s.al[id_i], sz_i = s.sz[id_i];
          const float bound_i = bound_s[warp * ROWS + i], best_before = best_c[i];
          const float row_least = fminf(bound_i, best_before);
          // Most pairs are far from the cheapest so far of either, and a product says so without the root: with
          // most = both - best - both / 2^20 positive and m2 <= most^2 (1 - 2^-20), the root is under `most` by more
          // than the roundings of all of these (a few 2^-24 of `both`), so the cost is above the best, and not a tie.
          // (That takes squares that are normal numbers: `most` is above 1e-15, and `slack` lets no pair through here in a
          // block whose norms may leave their range.) The lane's pairs of a row are looked at together: one branch for all.
          float m2[COLS], both[COLS];
          bool close[COLS], any = false;
#pragma unroll
          for (int j = 0; j < COLS; ++j) {
            m2[j] = __fadd_rn(__fadd_rn(sq_i, sq_j[j]), __fmul_rn(2.0f, acc[i][j]));
            both[j] = __fadd_rn(al_i, al_j[j]);
            const float most = fmaf(both[j], keep, -fmaxf(row_least, theirs_c[j]));
            close[j] = !(most > 1e-15f && m2[j] <= most * most * 0.99999904632568359375f);
            any = any || close[j];
          }
          if (any) {
#pragma unroll
            for (int j = 0; j < COLS; ++j) {
              if (!close[j] || id_j[j] < 0 || id_i == id_j[j] || __fadd_rn(sz_i, sz_j[j]) > p.bucket_cap) continue;
              const float whole = sqrtf(m2[j] > 0.0f ? m2[j] : 0.0f);
              const float cost = __fsub_rn(both[j], whole);
              if (cost < best_c[i] || (cost == best_c[i] && id_j[j] < best_j[i])) best_c[i] = cost, best_j[i] = id_j[j];
              // (the lists ascend, so a tie of two of this thread's rows stays with the first; one with what the partner knows
              // is settled where the minima are kept)
              if (cost < theirs_c[j] || (cost == theirs_c[j] && theirs_i[j] < 0)) theirs_c[j] = cost, theirs_i[j] = id_i;
            }
          }
          // (the lanes share what they found, so that in the next tile a pair is far from the cheapest of all of them; a local
          // block has few tiles a row)
          if (!LOCAL && __any_sync(0xffffffffu, best_c[i] < best_before && best_c[i] < bound_i)) {
            float least = best_c[i];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) least = fminf(least, __shfl_xor_sync(0xffffffffu, least, o));
            if (lane == 0) bound_s[warp * ROWS + i] = fminf(bound_i, least);
          }
        }
        __syncwarp();
#pragma unroll
        for (int j = 0; j < COLS; ++j)
          if (theirs_i[j] >= 0 && theirs_c[j] < INFINITY)
            atomicMin(mine + side * apart + id_j[j], pack_cheapest(theirs_c[j], theirs_i[j]));
      }
      if (my_rows <= 0) return;
      // The lanes fold a row's minima, halving the rows a lane holds while there is more than one: a lane ends up with
      // the minimum of the row its high bits number.
      int o = 16, my_row = 0;
#pragma unroll
      for (int n = ROWS; n > 1; n >>= 1, o >>= 1) {
        const bool upper = lane & o;
#pragma unroll
        for (int i = 0; i < n / 2; ++i) {
          const float give_c = upper ? best_c[i] : best_c[i + n / 2], keep_c = upper ? best_c[i + n / 2] : best_c[i];
          const int give_j = upper ? best_j[i] : best_j[i + n / 2], keep_j = upper ? best_j[i + n / 2] : best_j[i];
          const float c = __shfl_xor_sync(0xffffffffu, give_c, o);
          const int j = __shfl_xor_sync(0xffffffffu, give_j, o);
          const bool theirs = c < keep_c || (c == keep_c && j < keep_j);
          best_c[i] = theirs ? c : keep_c, best_j[i] = theirs ? j : keep_j;
        }
        my_row = 2 * my_row + (upper ? 1 : 0);
      }
      const int left = o;
#pragma unroll
      for (; o > 0; o >>= 1) {
        const float c = __shfl_xor_sync(0xffffffffu, best_c[0], o);
        const int j = __shfl_xor_sync(0xffffffffu, best_j[0], o);
        if (c < best_c[0] || (c == best_c[0] && j < best_j[0])) best_c[0] = c, best_j[0] = j;
      }
      if ((lane & (2 * left - 1)) == 0 && my_row < my_rows && best_c[0] < INFINITY)
        atomicMin(mine + side * apart + my_list[my_row], pack_cheapest(best_c[0], best_j[0]));
    };
    // This CTA's run of the tiles, a row tile at a time. A row tile meets the dirty partners from its own tile on.
    {
      const int all = (n_open + TILE - 1) / TILE, high = (n_dirty + TILE - 1) / TILE;
      // Eight rows a warp where that leaves every CTA a tile; else (a small block, a late round) two, for four times
      // the tiles. A last row tile of few rows gives every warp two or four of them. The last row tiles come first: where a CTA has
      // a block to itself, the rows that a later row tile meets have met their own by then, and know how cheap they are.
      constexpr int SMALL = kWardFewRows * kThreads / 32;
      const bool few = n_dirty <= SMALL || high * all - high * (high - 1) / 2 < ctas;
      const int height = few ? SMALL : TILE, row_tiles = (n_dirty + height - 1) / height;
      int64_t count = 0;
      for (int rt = 0; rt < row_tiles; ++rt) count += all - rt * height / TILE;
      const int64_t lo = count * rank / ctas, hi = count * (rank + 1) / ctas;
      int64_t before = 0;
      for (int rt = row_tiles - 1; rt >= 0 && before < hi; --rt) {
        const int own = rt * height / TILE, across = all - own, rows = n_dirty - rt * height;
        const int first = (int)max((int64_t)0, lo - before), end = (int)min((int64_t)across, hi - before);
        before += across;
        if (first >= end) continue;
        if (few || rows <= SMALL)
          search(std::integral_constant<int, kWardFewRows>(), rt * height, own + first, own + end);
        else if (rows <= 2 * SMALL)
          search(std::integral_constant<int, 2 * kWardFewRows>(), rt * height, own + first, own + end);
        else
          search(std::integral_constant<int, kWardRows>(), rt * height, own + first, own + end);
      }
    }
    everyone();
    if (gave_up) break;

    // ---- mutual cheapest pairs, held by their lower row; the cheapest of them merge, a tie to the lower row
    for (int i = tid; i < P; i += kThreads) {
      unsigned long long v = ~0ull;
      if (s.flag[i] & kOpen) {
        if (!LOCAL) {
          v = __ldcg(mine + side * apart + i);
        } else if (ctas == 1) {
          v = mine[i];
        } else {
#pragma unroll
          for (int c = 0; c < kWardMaxCtas; ++c)
            if (c < ctas) {
              const unsigned long long theirs = cluster.map_shared_rank(mine, c)[side * apart + i];
              v = theirs < v ? theirs : v;
            }
        }
      }
      s.cost[i] = v == ~0ull ? INFINITY : cheapest_cost(v);
      s.best[i] = v == ~0ull ? 0 : (uint16_t)(v & 0xFFFF);
    }
    if (tid == 0) n_merge_s = 0;
    __syncthreads();
    int n_pairs = 0;
    for (int i0 = 0; i0 < P; i0 += kThreads) {
      const int i = i0 + tid;
      const bool mutual = i < P && s.cost[i] < INFINITY && s.best[s.best[i]] == i && i < s.best[i];
      const unsigned votes = __ballot_sync(0xffffffffu, mutual);
      if (lane == 0) warp_count[warp] = __popc(votes);
      __syncthreads();
      int before = 0, all = 0;
#pragma unroll
      for (int w = 0; w < kThreads / 32; ++w) {
        if (w < warp) before += warp_count[w];
        all += warp_count[w];
      }
      if (mutual) s.pairs[n_pairs + before + __popc(votes & below)] = (uint16_t)i;
      n_pairs += all;
      __syncthreads();
    }
    const int merges_left = n_alive - p.bucket_count;
    for (int e = tid; e < n_pairs; e += kThreads) {
      const int i = s.pairs[e];
      if (n_pairs > merges_left) {
        const float ci = s.cost[i];
        int cheaper = 0;
        for (int f = 0; f < n_pairs; ++f) {
          const int j = s.pairs[f];
          cheaper += s.cost[j] < ci || (s.cost[j] == ci && j < i);
        }
        if (cheaper >= merges_left) continue;
      }
      // (pairs are disjoint: no row is another pair's)
      const int a = s.best[i];
      atomicAdd(&n_merge_s, 1);
      s.sz[i] = __fadd_rn(s.sz[i], s.sz[a]);
      s.parent[a] = (uint16_t)i;
      s.flag[i] |= kChanged | kMerged;
      s.flag[a] = kChanged;
      if (LOCAL || e % ctas == rank) {
        float4 row[D / 4];
#pragma unroll
        for (int k = 0; k < D / 4; ++k) {
          const float4 x = LOCAL ? *reinterpret_cast<const float4 *>(s.sums + (size_t)i * LD + 4 * k)
                                 : __ldcg(reinterpret_cast<const float4 *>(sums_g + (size_t)i * D + 4 * k));
          const float4 y = LOCAL ? *reinterpret_cast<const float4 *>(s.sums + (size_t)a * LD + 4 * k)
                                 : __ldcg(reinterpret_cast<const float4 *>(sums_g + (size_t)a * D + 4 * k));
          row[k] = make_float4(__fadd_rn(x.x, y.x), __fadd_rn(x.y, y.y), __fadd_rn(x.z, y.z), __fadd_rn(x.w, y.w));
        }
#pragma unroll
        for (int k = 0; k < D / 4; ++k)
          *reinterpret_cast<float4 *>(LOCAL ? s.sums + (size_t)i * LD + 4 * k : sums_g + (size_t)i * D + 4 * k) = row[k];
        const float q = row_square<D>(row), n = sqrtf(q > 0.0f ? q : 0.0f);
        if (LOCAL)
          s.sq[i] = q, s.al[i] = n;
        else
          sq_g[i] = q, al_g[i] = n;
      }
    }
    __syncthreads();
    if (n_merge_s == 0) break;
    n_alive -= n_merge_s;
    side ^= 1;
    make_lists();
    everyone();
    if (!LOCAL) {
      for (int e = tid; e < n_merged; e += kThreads) {
        const int i = s.merged[e];
        s.sq[i] = __ldcg(sq_g + i), s.al[i] = __ldcg(al_g + i);
      }
      __syncthreads();
    }
  }

  // Survivors numbered by their first pool; a merge keeps the lower pool, so a root is its bucket's first pool.
  __syncthreads();
  uint16_t *number = s.pairs;
  int numbered = 0;
  for (int i0 = 0; i0 < P; i0 += kThreads) {
    const int i = i0 + tid;
    const bool alive = i < P && (s.flag[i] & kAlive);
    const unsigned votes = __ballot_sync(0xffffffffu, alive);
    if (lane == 0) warp_count[warp] = __popc(votes);
    __syncthreads();
    int before = 0, all = 0;
#pragma unroll
    for (int w = 0; w < kThreads / 32; ++w) {
      if (w < warp) before += warp_count[w];
      all += warp_count[w];
    }
    if (alive) number[i] = (uint16_t)(numbered + before + __popc(votes & below));
    numbered += all;
    __syncthreads();
  }
  for (int i = rank * kThreads + tid; i < P; i += ctas * kThreads) {
    int r = i;
    while (s.parent[r] != r) r = s.parent[r];
    p.labels[g * P + i] = number[r];
  }
  if (rank == 0 && tid == 0) {
    p.reached[g] = n_alive <= p.bucket_count && !gave_up;
    if (p.rounds) p.rounds[g] = rounds;
  }
  if (LOCAL && ctas > 1) cluster.sync();  // (nobody's shared memory goes while another may still read it)
}

static size_t align_up(size_t n) { return (n + 255) & ~(size_t)255; }

static bool ward_is_local(int P, int d) { return P <= kWardLocalPools && d <= 64; }

bool ward_cluster_takes(int d) { return d == 16 || d == 32 || d == 64; }

size_t ward_cluster_workspace_bytes(int64_t G, int P, int d) {
  if (ward_is_local(P, d)) return 0;
  const size_t rows = (size_t)G * P;
  return align_up(rows * d * 4) + 2 * align_up(rows * 4) + align_up(2 * rows * 8) + (size_t)G * kWardApart * 4;
}

template <int D, bool LOCAL>
static int launch_ward(WardParams &p, int64_t G, cudaStream_t s) {
  // CTAs a block: as many as leave every block an SM a CTA, and two of the small tiles or more a CTA in the first round
  // (one block of 80 pools: 164 us with one CTA, 120 with five; 3 blocks of 256: 92 with four, 69 with eight). A local block
  // reads its cluster's shared memory, so it takes eight at most; a larger one has its rows and minima in the workspace, and
  // any number of CTAs can share it.
  constexpr int TILE = ward_tile(LOCAL), SMALL = TILE / kWardRows * kWardFewRows;
  const int64_t tiles = (int64_t)((p.P + TILE - 1) / TILE) * ((p.P + SMALL - 1) / SMALL);
  const int64_t most = tiles / 2 < sm_count() / G ? tiles / 2 : sm_count() / G;
  const int wanted = (int)(most < 1 ? 1 : most);
  int ctas = wanted < kWardMaxCtas ? wanted : kWardMaxCtas;
  WardShared<D, LOCAL> shared;
  const size_t smem = shared.carve(nullptr, p.P, ctas > 1);
  if (!allow_shared(ward_kernel<D, LOCAL>, shared.carve(nullptr, LOCAL ? kWardLocalPools : kWardMaxPools, true))) {
    (void)cudaGetLastError();
    return LSA_ERR_LAUNCH;
  }
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3((unsigned)(G * ctas)), config.blockDim = dim3(ward_threads(LOCAL));
  config.dynamicSmemBytes = smem, config.stream = s;
  cudaLaunchAttribute attribute[1];
  config.attrs = attribute, config.numAttrs = ctas > 1;
  attribute[0].id = cudaLaunchAttributeClusterDimension;
  attribute[0].val.clusterDim.y = attribute[0].val.clusterDim.z = 1;
  // (a cluster lives inside a GPC, and 148 SMs hold fewer clusters of eight than 18: one CTA less a block where a second
  // wave would follow)
  for (int fit = 0; ctas > 1; --ctas) {
    config.gridDim = dim3((unsigned)(G * ctas)), attribute[0].val.clusterDim.x = (unsigned)ctas;
    if (cudaOccupancyMaxActiveClusters(&fit, ward_kernel<D, LOCAL>, &config) != cudaSuccess) (void)cudaGetLastError();
    if (fit >= G) break;
  }
  attribute[0].val.clusterDim.x = (unsigned)ctas;
  // A larger block whose clusters leave SMs idle (16 blocks: six CTAs each, 96 of 148 SMs) takes a cooperative grid and a
  // counter in memory as its barrier. Pairings of clustered unit rows, one cluster a block -> the grid: one block of 4,096
  // buckets 2,322 -> 455 us, of 1,024 253 -> 159; 16 blocks of 4,096 3,124 -> 2,166 (those of an index of 1M tokens, which take
  // more rounds, 4,396 -> 3,066), of 640 no change. Of as many CTAs the cluster is the faster (its barrier
  // is: 32 blocks of 640 256 us, 268 as a grid), so it stays where it has them.
  if (LOCAL || wanted <= ctas) {
    p.arrived = nullptr;
  } else {
    ctas = wanted;
    config.numAttrs = 1;
    attribute[0].id = cudaLaunchAttributeCooperative;
    attribute[0].val.cooperative = 1;
    if (cudaMemsetAsync(p.arrived, 0, (size_t)G * kWardApart * 4, s) != cudaSuccess) return LSA_ERR_LAUNCH;
  }
  p.ctas = ctas;
  config.gridDim = dim3((unsigned)(G * ctas));
  (void)cudaLaunchKernelEx(&config, ward_kernel<D, LOCAL>, p);
  LSA_LAUNCH_CHECK();
  return LSA_OK;
}

int ward_cluster_run(const float *pool_keys, const float *pool_sizes, float uniform_size, int64_t G, int P, int d,
                     int bucket_count, float bucket_cap, int max_rounds, int64_t *labels, uint8_t *reached,
                     int32_t *rounds, void *workspace, cudaStream_t s) {
  WardParams p = {};
  p.pool_keys = pool_keys, p.pool_sizes = pool_sizes, p.uniform_size = uniform_size, p.bucket_cap = bucket_cap;
  p.P = P, p.bucket_count = bucket_count, p.max_rounds = max_rounds;
  p.labels = labels, p.reached = reached, p.rounds = rounds;
  const bool local = ward_is_local(P, d);
  if (!local) {
    const size_t rows = (size_t)G * P;
    unsigned char *at = (unsigned char *)workspace;
    p.sums = (float *)at, at += align_up(rows * d * 4);
    p.sq = (float *)at, at += align_up(rows * 4);
    p.al = (float *)at, at += align_up(rows * 4);
    p.cheapest = (unsigned long long *)at, at += align_up(2 * rows * 8);
    p.arrived = (int *)at;
  }
  if (d == 64) return local ? launch_ward<64, true>(p, G, s) : launch_ward<64, false>(p, G, s);
  if (d == 32) return local ? launch_ward<32, true>(p, G, s) : launch_ward<32, false>(p, G, s);
  return local ? launch_ward<16, true>(p, G, s) : launch_ward<16, false>(p, G, s);
}

}  // namespace lsa
