// Parameters shared by the prefill kernels and their host-side dispatcher.
#pragma once
#include "common.cuh"

namespace nvllm {

// Who stores packed rows: nobody, a warp that has nothing else to do, or from the key tiles in shared memory the epilogue
// warps, in blocks of three to an SM that warp.
enum class Store { None, Spare, Tiles };

// Where the key tiles of new rows are, for a prefill through the block table (prefill_route.cu).  Every cache block that
// new rows of a sequence lie in has a job: those of sequence b start at route_first_job(cu_q[b], b), in the order
// of its blocks.
struct RouteTables {
  int* tile_row = nullptr;  // [job][4]: first packed row of the 64-token tile, -1: read it through the table
  int* block = nullptr;     // [job]: its cache block, -1: none that is new as a whole
  int* source = nullptr;    // [sequence][max_blocks]: job of a cached block; anything, unless block[] agrees
  int jobs = 0;             // 0: no tables, everything is read in one place
};
constexpr int kRouteRagged = 1 << 30;  // in tile_row: the sequence ends inside the tile; rows for that sequence only
constexpr int kRouteJobs = 2048, kRouteEntries = 16384;  // the tables' sizes
constexpr int64_t kRouteJobBytes = 24 << 10;  // new rows of K and V per job from which on the tables are worth their launch
__host__ __device__ __forceinline__ int route_first_job(int q0, int b) { return (q0 >> 8) + 2 * b; }
inline int64_t route_jobs(int64_t n_new, int batch) { return (n_new >> 8) + 2 * static_cast<int64_t>(batch); }

struct PrefillParams {
  const __nv_bfloat16* q;
  int64_t q_stride;
  const __nv_bfloat16* k;  // packed K rows, or the K cache plane when block_tables != nullptr
  int64_t k_stride;
  const __nv_bfloat16* v;
  int64_t v_stride;
  const int32_t* block_tables;  // nullptr = packed K/V
  int64_t bt_stride;
  int max_blocks;
  __nv_bfloat16* out;
  int64_t out_stride;
  const int32_t* cu_q;
  const int32_t* cu_k;
  int batch, max_seqlen_q, max_seqlen_k;
  int hq, hkv, g, d;
  // persistent tcgen05 kernel only: query heads packed into one tile (1..8), its query tokens, 2^16 / heads
  int pack, tile_tokens, inv_pack;
  int spread_from;  // items above which a launch with no more of them than blocks, or of three blocks to an SM, takes the order of spread_item
  float scale_log2e;
  int64_t num_blocks;
  int* status;
  bool lengths_early;  // cu_q / cu_k were complete before the previous kernel in the stream let this one start
  // Packed rows that are also to be stored in the cache (slots nullptr: none): row i at slots[i].
  const int32_t* slots;
  __nv_bfloat16* k_store;
  __nv_bfloat16* v_store;
  int64_t n_new;
  Store store;  // persistent tcgen05 kernel only
  // and with a route: key and value are the packed rows, k and v the cache
  RouteTables route;
  const __nv_bfloat16* key;
  int64_t key_stride;
  const __nv_bfloat16* value;
  int64_t value_stride;
};

// Order of some launches: every q-th query tile of the list in turn, q the sequences' mean, so
// that all sequences' long tiles come first.  The item that the n-th draw of such a launch stands for; each of its
// items for one draw, which is what makes the launch complete whatever block draws when.
__host__ __device__ __forceinline__ int spread_item(int drawn, int n_tiles, int batch, int hgroups) {
  const int pi = drawn / hgroups, q = (n_tiles + batch - 1) / batch, full = n_tiles / q;
  const int rest = n_tiles - full * q, split = rest * (full + 1);
  const int col = pi < split ? pi / (full + 1) : rest + (pi - split) / full;
  const int row = pi - (pi < split ? col * (full + 1) : split + (col - rest) * full);
  return drawn + (row * q + col - pi) * hgroups;
}

// Sequences per launch of the persistent kernel (its per-sequence tables live in shared memory).
// The engine schedules at most 512 sequences per step (nanovllm/config.py:10).
constexpr int kPrefillMaxBatch = 1024;

// Warp-level mma.sync kernel: every supported geometry; cross-check, A/B baseline, and calls without a
// packed key row (batch <= 65535).
int launch_prefill_mma(const PrefillParams& p, cudaStream_t stream);
// tcgen05 / TMEM / TMA kernel in persistent blocks that pull (sequence, query tile, head) items
// from a global counter; batch <= kPrefillMaxBatch.  total_q / total_k bound the tiled loads.
int launch_prefill_tcp(const PrefillParams& p, int64_t total_q, int64_t total_k, cudaStream_t stream);
// How it is laid out on a device of `sms` multiprocessors: by the launch's sizes, whether there are rows to store (slots,
// n_new) and whether through the block table, with the route's tables or without (block_tables, route.jobs).
struct PrefillPlan {
  int blocks, grid;  // to an SM (three at head_dim 64 only), of the launch
  int pack;          // query heads in a tile
  int spread_from;   // see PrefillParams
  Store store;
};
PrefillPlan prefill_plan(const PrefillParams& p, int64_t total_q, int sms);
// Work items of such a launch at most.
int64_t prefill_max_items(int hq, int hkv, int max_seqlen_q, int batch);
// Fills the tables for a prefill through the block table and copies the rows that cannot be read packed.
int launch_prefill_route(const PrefillParams& p, RouteTables* tables, cudaStream_t stream);

}  // namespace nvllm
