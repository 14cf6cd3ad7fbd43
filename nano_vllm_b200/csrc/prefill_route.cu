// Where a prefill through the block table finds the rows of this step: the launch in front of it.
//
// The reference stores a step's rows and then reads everything through the table
// (nanovllm/layers/attention.py:62-73).  The rows of this step are also at hand packed, so the attention kernel can
// read them there, and write them to the cache from the key tiles that pass through its shared memory, instead of
// waiting for a copy of all of them (28 310 tokens of 8 KV heads: 38 us in front of 103).  This kernel says
// for each 64-token tile of new rows whether that gives what the table would: every row's slot must be the one
// that the table has for the row's position.  Rows for which it does not are copied here, as the store would.  A
// block that another sequence of the batch has as a cached block (prompts that share a prefix in one step) is told
// to that sequence, which then reads those packed rows.
//
// One thread block per cache block that new rows lie in (its "job"); bound by a chain of trips to memory: bounds of
// the sequences, table entry and slots, the other sequences' table entries.
#include <atomic>

#include "common.cuh"
#include "prefill.cuh"

namespace nvllm {

constexpr int kRouteLaunches = 32;  // that may be in flight at once
struct RouteScratch {
  int tile_row[kRouteJobs][4];
  int block[kRouteJobs];
  int source[kRouteEntries];
};
static __device__ RouteScratch g_route[kRouteLaunches];
static RouteScratch* g_route_addr[64] = {nullptr};

struct RouteParams {
  const uint4 *key, *value;
  int64_t key_stride16, value_stride16;  // in 16-byte pieces
  uint4 *k_cache, *v_cache;
  const int32_t *slots, *cu_q, *cu_k, *block_tables;
  int64_t bt_stride, n_new, num_blocks;
  int max_blocks, batch, per_row;  // per_row: 16-byte pieces of a row
  RouteTables out;
  int* status;
};

__global__ void __launch_bounds__(256) prefill_route_kernel(const RouteParams p) {
  pdl_wait();
  pdl_trigger();  // after the wait: the attention kernel that follows may read lengths and table early
  const int tid = threadIdx.x, job = blockIdx.x;
  const int64_t n_slots = p.num_blocks * kBlockSize;
  __shared__ int s_slot[kBlockSize];
  __shared__ int s_match[kBlockSize / 32];
  __shared__ int s_shared, s_twice;
  __shared__ int s_keys[kPrefillMaxBatch], s_cached[kPrefillMaxBatch];  // of every sequence

  auto copy_row = [&](int64_t row, int64_t slot, int piece) {
    p.k_cache[slot * p.per_row + piece] = __ldg(p.key + row * p.key_stride16 + piece);
    p.v_cache[slot * p.per_row + piece] = __ldg(p.value + row * p.value_stride16 + piece);
  };
  auto slot_of = [&](int64_t row) {
    const int64_t slot = p.slots[row];
    if (slot >= n_slots) atomicOr(p.status, NVLLM_STATUS_BAD_SLOT);
    return slot >= 0 && slot < n_slots ? static_cast<int>(slot) : -1;
  };
  // rows of no sequence: in front of the first and behind the last
  const int64_t front = p.cu_q[0], in_sequences = p.cu_q[p.batch] - front;
  for (int64_t r = job; r < p.n_new - in_sequences; r += gridDim.x) {
    const int64_t row = r < front ? r : r + in_sequences;
    const int slot = slot_of(row);
    for (int i = tid; slot >= 0 && i < p.per_row; i += 256) copy_row(row, slot, i);
  }

  // the job's sequence: the last one whose first job is not behind this one
  int before = 0;
  for (int b0 = 0; b0 < p.batch; b0 += 256) {
    const int b = b0 + tid;
    int q0 = 0;
    if (b < p.batch) {
      q0 = p.cu_q[b];
      s_keys[b] = p.cu_k[b + 1] - p.cu_k[b];
      s_cached[b] = s_keys[b] - (p.cu_q[b + 1] - q0);
    }
    before += __syncthreads_count(b < p.batch && route_first_job(q0, b) <= job);
  }
  int n = 0, x = -1, i = 0, q0 = 0, off = 0, lk = 0, b = before - 1;
  if (b >= 0) {
    q0 = p.cu_q[b], lk = s_keys[b], off = s_cached[b];
    i = (off >> 8) + job - route_first_job(q0, b);  // block of the sequence; negative where there are more queries than keys
    n = min((i + 1) * kBlockSize, lk) - max(i * kBlockSize, off);
  }
  if (n <= 0) {  // block-uniform
    if (tid < 4) p.out.tile_row[job * 4 + tid] = -1;
    if (tid == 4) p.out.block[job] = -1;
    return;
  }
  if (i >= 0 && i < p.max_blocks) x = p.block_tables[b * p.bt_stride + i];
  if (x >= p.num_blocks) x = -1;

  const int pos = i * kBlockSize + tid;
  const int64_t row = static_cast<int64_t>(q0) + pos - off;
  const bool is_new = pos >= off && pos < lk && row < p.n_new;
  const int slot = is_new ? slot_of(row) : -1;
  s_slot[tid] = slot;
  if (tid == 0) s_shared = s_twice = 0;
  // what lies behind the sequence's end need not match
  const int match = __all_sync(0xffffffffu, pos >= lk || (is_new && x >= 0 && slot == x * kBlockSize + tid));
  if ((tid & 31) == 0) s_match[tid >> 5] = match;
  __syncthreads();
  const bool whole = off >= 0 && i * kBlockSize >= off && x >= 0;  // no cached token in the block
  if (whole) {  // block-uniform
    // The table entries that are in use, of all sequences: eight lanes to a sequence, four sequences at a time.
    // Padding is not looked at: with whole rows 64 prompts of 100-1024 tokens took 149 us through a table 160 wide and
    // 140 through one 4 wide, 100 of 20-150 tokens 59 and 36; now 139 and 35.5 through either.
    for (int b0 = tid >> 3; b0 < p.batch; b0 += 128) {
      int used[4], most = 0;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        used[u] = b0 + 32 * u < p.batch ? min((s_keys[b0 + 32 * u] + kBlockSize - 1) / kBlockSize, p.max_blocks) : 0;
        most = max(most, used[u]);
      }
      for (int i2 = tid & 7; i2 < most; i2 += 8) {
        int entry[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) entry[u] = i2 < used[u] ? __ldg(p.block_tables + (b0 + 32 * u) * p.bt_stride + i2) : -1;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int b2 = b0 + 32 * u;
          if (entry[u] != x || (b2 == b && i2 == i)) continue;
          if (i2 * kBlockSize < s_cached[b2]) {
            p.out.source[b2 * p.max_blocks + i2] = job;
            s_shared = 1;
          } else {
            s_twice = 1;  // two sequences' new rows in one block: no telling whose rows it ends up with
          }
        }
      }
    }
  }
  __syncthreads();
  // A sequence's ragged end serves the sequence itself; for another one that has the block too it has to be in the cache.
  unsigned direct = 0;
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    const int first = i * kBlockSize + t * 64;
    const bool full = first + 64 <= lk;
    if (whole && !s_twice && first < lk && s_match[2 * t] && s_match[2 * t + 1] && (full || !s_shared)) direct |= 1u << t;
    if (tid == t) p.out.tile_row[job * 4 + t] = direct >> t & 1u ? static_cast<int>(q0 + first - off) | (full ? 0 : kRouteRagged) : -1;
  }
  if (tid == 4) p.out.block[job] = whole ? x : -1;
  for (int t = 0; t < 4; ++t) {
    const int first = i * kBlockSize + t * 64;
    if ((direct >> t & 1u) || first >= lk || first + 64 <= off) continue;
    for (int r = tid >> 5; r < 64; r += 8) {  // a row to a warp
      const int slot = s_slot[t * 64 + r];
      if (slot < 0) continue;
#pragma unroll 4
      for (int k = tid & 31; k < p.per_row; k += 32) copy_row(static_cast<int64_t>(q0) + first + r - off, slot, k);
    }
  }
}

int launch_prefill_route(const PrefillParams& p, RouteTables* tables, cudaStream_t stream) {
  static std::atomic<unsigned> launch_seq{0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
    (void)cudaGetLastError();
    return fail(NVLLM_E_NO_DEVICE, "prefill: no CUDA device is usable");
  }
  if (!g_route_addr[dev]) {
    void* at = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&at, g_route);
    if (e != cudaSuccess) return fail(NVLLM_E_CUDA, "prefill: set-up failed: %s", cudaGetErrorString(e));
    g_route_addr[dev] = static_cast<RouteScratch*>(at);
  }
  RouteScratch* s = g_route_addr[dev] + launch_seq.fetch_add(1) % kRouteLaunches;
  tables->tile_row = &s->tile_row[0][0];
  tables->block = s->block;
  tables->source = s->source;
  tables->jobs = static_cast<int>(route_jobs(p.n_new, p.batch));
  RouteParams r;
  r.key = reinterpret_cast<const uint4*>(p.key);
  r.value = reinterpret_cast<const uint4*>(p.value);
  r.key_stride16 = p.key_stride / 8;
  r.value_stride16 = p.value_stride / 8;
  r.k_cache = reinterpret_cast<uint4*>(p.k_store);
  r.v_cache = reinterpret_cast<uint4*>(p.v_store);
  r.slots = p.slots;
  r.cu_q = p.cu_q;
  r.cu_k = p.cu_k;
  r.block_tables = p.block_tables;
  r.bt_stride = p.bt_stride;
  r.n_new = p.n_new;
  r.num_blocks = p.num_blocks;
  r.max_blocks = p.max_blocks;
  r.batch = p.batch;
  r.per_row = p.hkv * p.d / 8;
  r.out = *tables;
  r.status = p.status;
  return launch_kernel("prefill (routes)", prefill_route_kernel, dim3(tables->jobs), dim3(256), 0, stream, r);
}

}  // namespace nvllm
