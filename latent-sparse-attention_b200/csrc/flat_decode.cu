// A decode step over a flat index in one call: the launches of lsa_index_map, lsa_flat_lists_at (past a top_p of 128
// lsa_visible_buckets, lsa_flat_select_decode and lsa_expand) and lsa_sparse_attend one after another, their intermediates in one
// workspace. On the GPU it is those calls; a host
// that makes them from an interpreter, with a dozen allocations between, takes longer over them than the GPU does.
#include "common.cuh"

namespace lsa {

// The workspace, carved in 256-byte pieces.
struct FlatDecodeRoom {
  float *index_queries, *lse;
  int32_t *visible, *picked, *lists, *lengths;
  int64_t *keys;
  void *select, *attend;
  size_t select_bytes, attend_bytes, total;

  FlatDecodeRoom(void *base, int64_t R, int Hq, int dh, int d_idx, int top_p, int64_t width, int select_splits, int splits) {
    total = 0;
    auto take = [&](size_t bytes) {
      unsigned char *p = (unsigned char *)base + total;
      total += (bytes + 255) & ~(size_t)255;
      return (void *)p;
    };
    select_bytes = lsa_flat_lists_at_workspace_bytes(R, top_p, select_splits);
    attend_bytes = lsa_sparse_attend_workspace_bytes(R, Hq, dh, splits);
    index_queries = (float *)take((size_t)R * d_idx * 4), lse = (float *)take((size_t)R * Hq * 4);
    visible = (int32_t *)take((size_t)R * 4), picked = (int32_t *)take((size_t)R * top_p * 4);
    lists = (int32_t *)take((size_t)R * width * 4), lengths = (int32_t *)take((size_t)R * 4);
    keys = (int64_t *)take((size_t)R * top_p * 8);
    select = take(select_bytes), attend = take(attend_bytes);
  }
};

}  // namespace lsa

LSA_API size_t lsa_flat_decode_workspace_bytes(int64_t R, int Hq, int dh, int d_idx, int top_p, int64_t width, int select_splits,
                                               int splits) {
  if (R <= 0 || Hq <= 0 || dh <= 0 || d_idx <= 0 || top_p <= 0 || width <= 0) return 0;
  return lsa::FlatDecodeRoom(nullptr, R, Hq, dh, d_idx, top_p, width, select_splits, splits).total;
}

LSA_API int lsa_flat_decode(const uint16_t *q, int64_t R, int Hq, int dh, int64_t q_row_stride, int64_t q_head_stride,
                            const void *map, int map_dtype, int dh_off, int dh_used, int d_idx, const int64_t *positions,
                            const float *centroids, int64_t m, const int32_t *members, int bucket_cap, int64_t block,
                            int64_t block_buckets, int top_p, int top_k, int sink, int window, int select_splits,
                            const uint16_t *k, const uint16_t *v, int64_t slots, int Hkv, int64_t kv_row_stride,
                            int64_t kv_head_stride, float scale, int splits, uint16_t *out_bf16, int32_t *expand_status,
                            void *workspace, size_t workspace_bytes, void *stream) {
  LSA_REQUIRE(q && map && positions && k && v && out_bf16 && workspace, LSA_ERR_NULL);
  LSA_REQUIRE(R >= 0 && Hq >= 1 && Hkv >= 1 && Hq % Hkv == 0 && dh >= 1 && d_idx >= 1 && top_p >= 1 && top_k >= 1 && sink >= 0 &&
                  window >= 1 && select_splits >= 1 && splits >= 1,
              LSA_ERR_ARGUMENT);
  if (R == 0) return LSA_OK;
  const int64_t width = (int64_t)top_k + window + sink;
  const lsa::FlatDecodeRoom room(workspace, R, Hq, dh, d_idx, top_p, width, select_splits, splits);
  LSA_REQUIRE(workspace_bytes >= room.total, LSA_ERR_WORKSPACE);
  int rc = lsa_index_map(q, LSA_DTYPE_BF16, R, Hq, Hq / Hkv, dh_off, dh_used, q_row_stride, q_head_stride, map, map_dtype, d_idx, 1,
                         room.index_queries, nullptr, stream);
  const bool at = top_p <= 128;  // (the scan finds what its rows see by itself, and leaves lists; a layer makes no other call)
  if (rc == LSA_OK && at)
    rc = lsa_flat_lists_at(room.index_queries, R, d_idx, centroids, positions, block, block_buckets, m, members, bucket_cap, top_p,
                           top_k, sink, window, select_splits, room.lists, room.lengths, room.select, room.select_bytes, stream);
  if (rc == LSA_OK && !at) rc = lsa_visible_buckets(positions, R, block, block_buckets, m, room.visible, stream);
  if (rc == LSA_OK && !at)
    rc = lsa_flat_select_decode(room.index_queries, R, d_idx, centroids, nullptr, room.visible, top_p, select_splits, room.keys,
                                room.picked, room.select, room.select_bytes, stream);
  if (rc == LSA_OK && !at)
    rc = lsa_expand(room.picked, R, top_p, positions, members, m, bucket_cap, nullptr, nullptr, top_k, sink, window, nullptr, 0, 0,
                    INT64_MAX, 1, 1, 0, LSA_EXPAND_NO_PAD, room.lists, room.lengths, expand_status, stream);
  if (rc == LSA_OK)
    rc = lsa_sparse_attend(q, R, Hq, dh, q_row_stride, q_head_stride, k, v, slots, 0, Hkv, kv_row_stride, kv_head_stride, room.lists,
                           width, room.lengths, nullptr, nullptr, scale, splits, out_bf16, nullptr, room.lse, room.attend,
                           room.attend_bytes, stream);
  return rc;
}
