// nvllm_prefill_varlen: argument checks and kernel selection.
#include <cstdlib>

#include "common.cuh"
#include "prefill.cuh"

namespace nvllm {

// The persistent tcgen05 kernel is the product.  NVLLM_PREFILL_IMPL=mma (read on every call)
// selects the warp-level mma.sync kernel instead: the cross-check of the tests and the A/B
// baseline of measurements, chosen by the library itself only for packed keys of no rows, of which
// no tensor map can be made.
static bool forced_mma() {
  const char* forced = std::getenv("NVLLM_PREFILL_IMPL");
  return forced && forced[0] == 'm';
}

static int prefill_common(const void* q, int64_t q_row_stride, const void* k, int64_t k_row_stride, const void* v,
                          int64_t v_row_stride, const int32_t* block_tables, int64_t bt_row_stride, int32_t max_blocks, void* out,
                          int64_t out_row_stride, const int32_t* cu_seqlens_q, const int32_t* cu_seqlens_k, int64_t total_q,
                          int64_t total_k, int32_t batch, int32_t max_seqlen_q, int32_t max_seqlen_k, int32_t num_q_heads,
                          int32_t num_kv_heads, int32_t head_dim, float scale, int64_t num_blocks, void* stream,
                          bool lengths_early, const int32_t* slots, void* k_store, void* v_store, const void* key = nullptr,
                          int64_t key_row_stride = 0, const void* value = nullptr, int64_t value_row_stride = 0) {
  if (head_dim != 64 && head_dim != 128)
    return fail(NVLLM_E_GEOMETRY, "prefill_varlen: head_dim=%d unsupported (64 or 128)", head_dim);
  if (num_q_heads <= 0 || num_kv_heads <= 0 || num_q_heads % num_kv_heads)
    return fail(NVLLM_E_GEOMETRY, "prefill_varlen: Hq=%d must be a positive multiple of Hkv=%d", num_q_heads, num_kv_heads);
  if (batch < 0 || num_q_heads > 65535)
    return fail(NVLLM_E_GEOMETRY, "prefill_varlen: batch=%d / Hq=%d outside the launch limits", batch, num_q_heads);
  if (max_seqlen_q < 0 || max_seqlen_k < 0)
    return fail(NVLLM_E_GEOMETRY, "prefill_varlen: negative max_seqlen");
  if (total_q < 0 || total_k < 0) return fail(NVLLM_E_GEOMETRY, "prefill_varlen: negative total_q / total_k");
  if (batch == 0 || max_seqlen_q == 0 || total_q == 0) return NVLLM_OK;
  if (!q || !k || !v || !out || !cu_seqlens_q || !cu_seqlens_k)
    return fail(NVLLM_E_NULL, "prefill_varlen: NULL pointer argument");
  const int64_t qrow = static_cast<int64_t>(num_q_heads) * head_dim;
  const int64_t kvrow = static_cast<int64_t>(num_kv_heads) * head_dim;
  if (q_row_stride < qrow || out_row_stride < qrow)
    return fail(NVLLM_E_GEOMETRY, "prefill_varlen: q/out row stride smaller than Hq*D");
  if (q_row_stride % 8 || out_row_stride % 8 || !aligned16(q) || !aligned16(out) || !aligned16(k) || !aligned16(v))
    return fail(NVLLM_E_ALIGN, "prefill_varlen: pointers and row strides must be 16-byte aligned");
  if (block_tables) {
    if (max_blocks <= 0 || bt_row_stride < max_blocks || num_blocks <= 0)
      return fail(NVLLM_E_GEOMETRY, "prefill_varlen: paged mode needs max_blocks>0, bt_row_stride>=max_blocks, num_blocks>0");
  } else {
    if (k_row_stride < kvrow || v_row_stride < kvrow)
      return fail(NVLLM_E_GEOMETRY, "prefill_varlen: k/v row stride smaller than Hkv*D");
    if (k_row_stride % 8 || v_row_stride % 8)
      return fail(NVLLM_E_ALIGN, "prefill_varlen: k/v row strides must be multiples of 8 elements");
  }
  const bool has_rows = block_tables || total_k > 0;
  const bool use_mma = forced_mma() || !has_rows;
  if (!use_mma && batch > kPrefillMaxBatch)
    return fail(NVLLM_E_GEOMETRY, "prefill_varlen: batch=%d exceeds the %d sequences of one launch", batch, kPrefillMaxBatch);
  if (batch > 65535) return fail(NVLLM_E_GEOMETRY, "prefill_varlen: batch=%d outside the launch limits", batch);
  PrefillParams p;
  p.status = status_word();
  if (!p.status) return fail(NVLLM_E_NO_DEVICE, "prefill_varlen: no CUDA device is usable");
  p.q = static_cast<const __nv_bfloat16*>(q);
  p.q_stride = q_row_stride;
  p.k = static_cast<const __nv_bfloat16*>(k);
  p.k_stride = k_row_stride;
  p.v = static_cast<const __nv_bfloat16*>(v);
  p.v_stride = v_row_stride;
  p.block_tables = block_tables;
  p.bt_stride = bt_row_stride;
  p.max_blocks = max_blocks;
  p.out = static_cast<__nv_bfloat16*>(out);
  p.out_stride = out_row_stride;
  p.cu_q = cu_seqlens_q;
  p.cu_k = cu_seqlens_k;
  p.batch = batch;
  p.max_seqlen_q = max_seqlen_q;
  p.max_seqlen_k = max_seqlen_k;
  p.hq = num_q_heads;
  p.hkv = num_kv_heads;
  p.g = num_q_heads / num_kv_heads;
  p.d = head_dim;
  p.pack = 1;
  p.scale_log2e = scale * 1.4426950408889634f;
  p.num_blocks = num_blocks;
  p.lengths_early = lengths_early;
  p.slots = slots;
  p.k_store = static_cast<__nv_bfloat16*>(k_store);
  p.v_store = static_cast<__nv_bfloat16*>(v_store);
  p.n_new = slots ? total_k : 0;
  if (key) {  // the rows of a prefill through the table
    p.key = static_cast<const __nv_bfloat16*>(key);
    p.key_stride = key_row_stride;
    p.value = static_cast<const __nv_bfloat16*>(value);
    p.value_stride = value_row_stride;
    const int rc = launch_prefill_route(p, &p.route, static_cast<cudaStream_t>(stream));
    if (rc) return rc;
  }
  if (use_mma) return launch_prefill_mma(p, static_cast<cudaStream_t>(stream));
  return launch_prefill_tcp(p, total_q, total_k, static_cast<cudaStream_t>(stream));
}

}  // namespace nvllm

extern "C" int nvllm_prefill_varlen(const void* q, int64_t q_row_stride, const void* k, int64_t k_row_stride,
                                    const void* v, int64_t v_row_stride, const int32_t* block_tables,
                                    int64_t bt_row_stride, int32_t max_blocks, void* out, int64_t out_row_stride,
                                    const int32_t* cu_seqlens_q, const int32_t* cu_seqlens_k, int64_t total_q,
                                    int64_t total_k, int32_t batch, int32_t max_seqlen_q, int32_t max_seqlen_k, int32_t num_q_heads,
                                    int32_t num_kv_heads, int32_t head_dim, float scale, int64_t num_blocks,
                                    void* stream) {
  return nvllm::prefill_common(q, q_row_stride, k, k_row_stride, v, v_row_stride, block_tables, bt_row_stride, max_blocks, out,
                               out_row_stride, cu_seqlens_q, cu_seqlens_k, total_q, total_k, batch, max_seqlen_q, max_seqlen_k,
                               num_q_heads, num_kv_heads, head_dim, scale, num_blocks, stream, false, nullptr, nullptr, nullptr);
}

extern "C" int nvllm_prefill_item(int32_t drawn, int32_t query_tiles, int32_t batch, int32_t head_groups) {
  using namespace nvllm;
  if (batch <= 0 || query_tiles <= 0 || head_groups <= 0 || drawn < 0 || drawn >= static_cast<int64_t>(query_tiles) * head_groups)
    return fail(NVLLM_E_GEOMETRY, "prefill_item: drawn=%d query_tiles=%d batch=%d head_groups=%d invalid", drawn, query_tiles, batch, head_groups);
  return spread_item(drawn, query_tiles, batch, head_groups);
}

extern "C" int nvllm_prefill_plan(int64_t total_q, int64_t total_k, int32_t batch, int32_t max_seqlen_q, int32_t max_seqlen_k,
                                  int32_t num_q_heads, int32_t num_kv_heads, int32_t head_dim, int32_t rows, int32_t num_sms,
                                  int32_t* blocks_per_sm, int32_t* reordered_from, int32_t* store) {
  using namespace nvllm;
  if (head_dim != 64 && head_dim != 128) return fail(NVLLM_E_GEOMETRY, "prefill_plan: head_dim=%d unsupported (64 or 128)", head_dim);
  if (num_q_heads <= 0 || num_kv_heads <= 0 || num_q_heads % num_kv_heads || batch <= 0 || total_q <= 0 || total_k < 0 ||
      max_seqlen_q <= 0 || max_seqlen_k < 0 || rows < 0 || rows > 3 || num_sms <= 0)
    return fail(NVLLM_E_GEOMETRY, "prefill_plan: Hq=%d Hkv=%d batch=%d total_q=%lld rows=%d num_sms=%d invalid", num_q_heads, num_kv_heads,
                batch, (long long)total_q, rows, num_sms);
  if (!blocks_per_sm || !reordered_from || !store) return fail(NVLLM_E_NULL, "prefill_plan: NULL pointer argument");
  PrefillParams p{};
  p.batch = batch;
  p.max_seqlen_q = max_seqlen_q;
  p.max_seqlen_k = max_seqlen_k;
  p.hq = num_q_heads;
  p.hkv = num_kv_heads;
  p.g = num_q_heads / num_kv_heads;
  p.d = head_dim;
  const bool stored = rows == 1 || rows == 2;
  p.slots = stored ? store : nullptr;  // these two are only asked for whether there are any
  p.block_tables = rows >= 2 ? store : nullptr;
  p.n_new = stored ? total_k : 0;
  p.route.jobs = rows == 2;
  const PrefillPlan plan = prefill_plan(p, total_q, num_sms);
  *blocks_per_sm = plan.blocks;
  *reordered_from = plan.spread_from;
  *store = static_cast<int32_t>(plan.store);
  return NVLLM_OK;
}

extern "C" int nvllm_attention_prefill(const void* q, int64_t q_row_stride, const void* key, int64_t key_row_stride,
                                       const void* value, int64_t value_row_stride, const int32_t* slot_mapping, void* k_cache,
                                       void* v_cache, const int32_t* block_tables, int64_t bt_row_stride, int32_t max_blocks,
                                       void* out, int64_t out_row_stride, const int32_t* cu_seqlens_q,
                                       const int32_t* cu_seqlens_k, int64_t total_q, int64_t total_k, int32_t batch,
                                       int32_t max_seqlen_q, int32_t max_seqlen_k, int32_t num_q_heads, int32_t num_kv_heads,
                                       int32_t head_dim, float scale, int64_t num_blocks, void* stream) {
  using namespace nvllm;
  // Packed keys do not depend on the cache: warps of the prefill that have nothing else to do copy them
  // there.  Through the table the copy has to be complete first; the lengths are then ranked under it.
  const bool inside = !block_tables && batch > 0 && max_seqlen_q > 0 && total_q > 0 && total_k > 0 && !forced_mma() &&
                      total_k * num_kv_heads * head_dim / 8 < (1ll << 30);  // indexed with 32 bits
  // Or, where blocks work on several items one after the other, they read this step's rows packed too and store them on the
  // way, with the tables of prefill_route.cu: 64 prompts of 100-1024 tokens, some with cached prefixes, 16 / 8 heads
  // 161 -> 140 us (chain of three inputs), 8 of 1500-2048 114 -> 105, 8 of 100-1024 27.1 -> 24.4, whatever the table's width.
  // With an item to a block the copy is the shorter way (4 prompts of 300-400 tokens 15.6, 16.0 with the tables).  So it
  // is where the tables' blocks have few bytes each to save: at 4 / 2 heads of 128, 100 prompts of 20-150 tokens (36 KB a
  // block) gain 10 %, 200 of 30-100 (29) 1 %, 256 of 20-64 (19) lose 7 %, 400 of 10-40 (12) 9 %; at 14 / 2 heads of 64, 64 of
  // 100-1024 (63) gain 0.4 %, 100 of 20-150 (18) lose 1 %, 200 of 30-100 (15) 6 %; at 7 / 1 and 8 / 1 heads the sign changes
  // between 15 and 30 too.
  const bool routed = block_tables && batch > 0 && batch <= kPrefillMaxBatch && max_blocks > 0 && !forced_mma() && total_q > 0 &&
                      max_seqlen_q > 0 && total_k >= total_q && total_k < kRouteRagged && route_jobs(total_k, batch) <= kRouteJobs &&
                      static_cast<int64_t>(batch) * max_blocks <= kRouteEntries && num_kv_heads > 0 && num_q_heads > 0 &&
                      num_q_heads % num_kv_heads == 0 &&
                      total_k * num_kv_heads * head_dim * 4 >= kRouteJobBytes * route_jobs(total_k, batch) &&
                      prefill_max_items(num_q_heads, num_kv_heads, max_seqlen_q, batch) > 2 * num_sms();
  const int rc = store_kvcache(!inside && !routed, key, key_row_stride, value, value_row_stride, k_cache, v_cache, slot_mapping, total_k,
                               num_kv_heads * head_dim, num_blocks * kBlockSize, stream);
  if (rc) return rc;
  return prefill_common(q, q_row_stride, block_tables ? k_cache : key, key_row_stride, block_tables ? v_cache : value,
                        value_row_stride, block_tables, bt_row_stride, max_blocks, out, out_row_stride, cu_seqlens_q, cu_seqlens_k,
                        total_q, total_k, batch, max_seqlen_q, max_seqlen_k, num_q_heads, num_kv_heads, head_dim, scale, num_blocks,
                        stream, !inside && total_k > 0, inside || routed ? slot_mapping : nullptr, k_cache, v_cache,
                        routed ? key : nullptr, key_row_stride, value, value_row_stride);
}
