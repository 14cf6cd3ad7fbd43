// Varlen causal GQA prefill on the 5th-generation tensor cores (tcgen05 + TMEM + TMA), head_dim
// 64 or 128.  Math follows the prefill branch of nanovllm/layers/attention.py:67-73
// (flash_attn_varlen_func, causal, optional block table).
//
// Tile pipeline: 128 query rows x 64-key tiles; S = Q K^T (SS form, both operands K-major in
// shared memory) into one of two S buffers in TMEM; the softmax warps (thread = query row) read
// their row of S with tcgen05.ld, write P as packed bf16 over it (three blocks to an SM: one S buffer, P
// beside it) with tcgen05.st; O += P V (TS
// form: P from TMEM, V as an MN-major shared-memory operand); Q, K, V arrive by TMA tile loads
// (128-byte swizzle, no multicast) into a two-stage ring; one tcgen05.commit per MMA group.
// Two forms, see Geo and three_blocks: two blocks of twelve warps to an SM, which the following describes, or at head_dim 64
// three of eight, without the epilogue warps: there the softmax warps write an item's results and the copy warp stores rows
// from the key tiles.
// Twelve warps: 0-3 softmax / correction (thread = query row), 4-7 epilogue (same rows: when an
// item's last P V product is done they normalise O and store it while the softmax warps are
// already in the next item's first tile, and write packed K/V rows to the cache from the key tiles), warp 8 = TMA producer of
// Q and K, warp 9 = MMA issuer, warp 10 = TMA producer of V (one elected lane each), warp 11 = a copy of rows that no
// tile stores; the three warp groups trade registers at start-up (setmaxnreg) so that two such blocks fit an
// SM.  A thread block does not end with its query tile: two blocks per SM stay resident
// for the whole launch, keep their TMEM allocation and barriers, and pull work items (sequence,
// query tile, head group) from a global counter.  Under grouped-query attention the 128 rows of a tile are
// 128/n tokens x n query heads that share a KV head (n = 1, 2, 4 or 8), not 128 tokens of one
// head: the causal diagonal and the ragged end of a sequence then cut through a narrower band
// of tokens, so fewer of the issued products are masked or padding.  What this buys on short prompts, where a block only has a handful of
// key tiles: the block launch / TMEM allocation / barrier set-up is paid once, the producer
// lane fetches the next item and starts its Q and first K loads while the current item is
// still in its last softmax, and the tensor pipe runs the next item's first S product under
// the current item's epilogue.
//
// Order of the items: sequences longest first (ranked in shared memory by every block at start-up,
// for batches of up to SORT_BATCH sequences), a sequence's long tiles first, head groups fastest.
// The blocks that are still busy when the counter runs out are then working on the cheapest
// items, so the launch ends without a tail of half-idle SMs.  At head_dim 128 where there are no more items than blocks, of
// prompts of about one length, and with three blocks to an SM where prompts have the same number of query tiles, all
// sequences' long tiles go first instead.
//
// Item hand-off: the producer lane decodes an item into one of two descriptor slots in shared
// memory (ITEM_FULL / ITEM_FREE barriers).  All rings keep running across items: tile t of the
// block's life uses stage t&1 and barrier phase (t>>1)&1, so the next item's first K/V tiles
// are fetched under the current item's last products.  The first P V product of an item waits
// for the previous item's O to be read (O_FREE; by the softmax warps themselves where there are no others); the softmax
// warps leave each row's 1 / sum in shared memory (EPI_FULL) and move on.  The epilogue needs no block-wide buffer: an epilogue
// warp owns the same 32 rows in TMEM and in the output, and passes them 32 columns at a time
// through a private 2 KB patch of shared memory to turn row-per-lane registers into 64-byte row
// segments.
//
// Code size: the warps of a block run seven different loops at the same time, and what they have to fetch of them
// is on the path of each: in a kernel of 84 KB (loops unrolled as the compiler likes, barrier waits of 25
// instructions, barriers set up one after the other by one thread) every fifth cycle of a warp waited for
// instructions.  Hence the loops that are kept rolled here, the short wait, and no division for a row's token: 57-59 KB;
// one prompt of 201 tokens 9.5 -> 9.05 us, of 1000 19.1 -> 18.1, 64 of 100-1024 tokens 136 -> 123.
#include <algorithm>
#include <atomic>
#include <cstdlib>

#include "common.cuh"
#include "prefill.cuh"
#include "prefill_tc.cuh"
#include "sm100.cuh"

namespace nvllm {
using namespace sm100;

namespace tcp {
using namespace tc;
constexpr int MAX_BATCH = kPrefillMaxBatch;  // prefix array of query tiles per sequence lives in shared memory
constexpr int SORT_BATCH = 256;  // batches up to this size are ranked by length (B^2 / 192 compares per thread)
enum PBar {
  ITEM_FULL0 = tc::NUM_BARS, ITEM_FULL1, ITEM_FREE0, ITEM_FREE1, O_FREE, EPI_FULL0, EPI_FULL1,
  K_DUE0, K_DUE1, V_DUE0, V_DUE1, K_STORED0, K_STORED1, V_STORED0, V_STORED1, P_NUM_BARS,
  S_FREE = O_FREE  // blocks of two groups have this one and not the other
};
constexpr int REGS_LAUNCH = 80;  // a thread's at launch, in every form: 768 threads an SM
// Shared-memory layout and tile sizes for one head_dim (64 or 128).  A tile row is split into
// 64-element (128-byte) sub-tiles, the unit of the 128-byte swizzle.
template <int D_, bool TRIO_>
struct Geo {
  static constexpr int D = D_;
  static constexpr int NSUB = D / 64;               // sub-tiles per tile row
  static constexpr int Q_SUB = BM * 128, Q_BYTES = NSUB * Q_SUB;
  static constexpr int KV_SUB = BN * 128, KV_BYTES = NSUB * KV_SUB;
  static constexpr int OFF_Q = 0, OFF_K = Q_BYTES, OFF_V = OFF_K + KST * KV_BYTES;
  static constexpr int OFF_STAGE = OFF_V + KST * KV_BYTES;  // 4 warps x 32 rows x 64 B of output
  static constexpr int OFF_CTRL = OFF_STAGE + 4 * 2048;     // barriers (8 B each)
  static constexpr int OFF_SLOTS = OFF_CTRL + 256;         // two item descriptors of 8 ints
  static constexpr int OFF_MISC = OFF_SLOTS + 64;          // tmem address, abort flag
  static constexpr int OFF_PREFIX = OFF_MISC + 64;         // (MAX_BATCH + 1) ints
  static constexpr int OFF_ORDER = OFF_PREFIX + (MAX_BATCH + 1) * 4 + 60;  // MAX_BATCH u16: sequences, longest first
  static constexpr int OFF_INV = OFF_ORDER + MAX_BATCH * 2;  // 2 items x 128 rows: 1 / row sum, softmax -> epilogue
  static constexpr int SMEM = OFF_INV + 2 * 128 * 4 + 1024;
  static constexpr int OCH = D / 32;      // 32-column chunks of O
  static constexpr int ROWB = D * 2;      // bytes of one output row
  static constexpr int PIECES = D / 8;    // 16-byte pieces of one row
  // A block's warps in groups of four: softmax, epilogue, and (producer of Q and K, MMA issuer, producer of V, copy).
  // Registers are handed over between the groups at start-up (setmaxnreg): the softmax rows need about twice what a
  // thread has at launch, the other groups a fraction.
  // TRIO, at head_dim 64: no epilogue group, and three blocks to an SM instead of two.  A softmax warp takes 1650 cycles
  // for a tile (300 of them waiting for S) whose exponentials are 512 of its scheduler's and whose products 300 of the
  // tensor pipe: two of them keep a scheduler's exponentials busy for 66 % of the time, three for 70-80.  A block has 160
  // columns of TMEM: S 64, O 64 and P 32 (two blocks: P over the scores, of which there are two).  Scores and P in places
  // of their own in two blocks made them slower (4 prompts of 4096 tokens 180 -> 206 us), as did steps of two key tiles
  // (197); rings of four stages, or the row maximum beside the exponentials instead of in front of them, nothing.
  static constexpr bool TRIO = TRIO_;
  static constexpr int BLOCKS = TRIO ? 3 : 2, NTHREADS = TRIO ? 256 : 384, FIRST_OTHER = TRIO ? 4 : 8;
  static constexpr int REGS_SOFTMAX = TRIO ? 104 : 136, REGS_EPILOGUE = TRIO ? 0 : 64, REGS_OTHER = TRIO ? 56 : 40;
  static_assert(128 * (REGS_SOFTMAX + REGS_EPILOGUE + REGS_OTHER) <= NTHREADS * REGS_LAUNCH, "register pool of a block");
  static constexpr int TMEM_O = TRIO ? 64 : 128;  // column of O
};
constexpr int NUM_SLOTS = 64;                     // launches that may be in flight at once
static_assert(P_NUM_BARS * 8 <= 256, "barrier area");
}  // namespace tcp

// Work counters, one pair per launch slot; the last block of a launch to leave resets its pair.
__device__ unsigned int g_item_counter[tcp::NUM_SLOTS];
__device__ unsigned int g_done_counter[tcp::NUM_SLOTS];

struct Item {
  int b, h, m0, q0, Lq, k0, Lk, n_kv;  // n_kv < 0: no more work
};

// Key tiles that the first `tokens` query tokens of a sequence see.
__device__ __forceinline__ int key_tiles(int tokens, int Lq, int Lk) {
  const int end = min(Lk, min(tokens, Lq) + (Lk - Lq));
  return end > 0 ? (end + tc::BN - 1) / tc::BN : 0;
}
// Key tiles below this one are also seen by an item before this one in its sequence and are stored there;
// of the items that share a KV head's tiles only the first group of query heads stores.
__device__ __forceinline__ int first_stored(const Item& x, int g) {
  return x.h % g == 0 ? (x.m0 > 0 ? key_tiles(x.m0, x.Lq, x.Lk) : 0) : x.n_kv;
}

template <int D, bool ROUTED, bool TRIO>
__global__ void __launch_bounds__(tcp::Geo<D, TRIO>::NTHREADS, tcp::Geo<D, TRIO>::BLOCKS)
prefill_tcp_kernel(const PrefillParams p, const __grid_constant__ CUtensorMap tmap_q,
                   const __grid_constant__ CUtensorMap tmap_k, const __grid_constant__ CUtensorMap tmap_v,
                   const __grid_constant__ CUtensorMap tmap_key, const __grid_constant__ CUtensorMap tmap_value,
                   const int counter_slot) {
  using namespace tcp;
  using G = Geo<D, TRIO>;
  constexpr int Q_SUB = G::Q_SUB, KV_BYTES = G::KV_BYTES, KV_SUB = G::KV_SUB;
  constexpr int OFF_Q = G::OFF_Q, OFF_K = G::OFF_K, OFF_V = G::OFF_V, OFF_CTRL = G::OFF_CTRL;
  constexpr int OFF_SLOTS = G::OFF_SLOTS, OFF_MISC = G::OFF_MISC, OFF_PREFIX = G::OFF_PREFIX, OFF_ORDER = G::OFF_ORDER;
  constexpr int OCH = G::OCH, PIECES = G::PIECES, NTHREADS_P = G::NTHREADS;
  constexpr int W_QK = G::FIRST_OTHER, W_MMA = W_QK + 1, W_V = W_QK + 2;
  extern __shared__ unsigned char smem_raw[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  unsigned char* base_ptr = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t bars = base + OFF_CTRL;
  auto bar = [&](int i) { return bars + 8u * i; };
  volatile int* slots = reinterpret_cast<volatile int*>(base_ptr + OFF_SLOTS);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(base_ptr + OFF_MISC);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(base_ptr + OFF_MISC + 8);
  int* prefix = reinterpret_cast<int*>(base_ptr + OFF_PREFIX);  // prefix[i] = query tiles before the i-th sequence in order
  unsigned short* order = reinterpret_cast<unsigned short*>(base_ptr + OFF_ORDER);  // order[i] = i-th longest sequence
  // Head packing: the rows of a tile are BMT = 128 / n query tokens x n query heads of one KV head
  // (row = token * n + head; n = p.pack need not be a power of two: 7 heads x 18 tokens leave two
  // rows unused), so short and ragged sequences waste fewer rows above the diagonal and past
  // their end, and the packed heads share every K/V tile.
  constexpr int TILES = kBlockSize / BN;  // key tiles of a cache block
  const int pack = p.pack, BMT = p.tile_tokens;
  auto token_of = [&](int row) { return row * p.inv_pack >> 16; };  // row / pack, row < 128

  pdl_trigger();
  if (warp == W_MMA && lane < P_NUM_BARS) {  // a barrier per lane
    // four softmax warps fill P and the normalisers; four epilogue warps free O and store rows; an item slot is
    // free when the softmax warps, the epilogue warps, the MMA issuer and the V producer are done with it.  Two groups:
    // the softmax warps free S, the last warp stores rows and has to do with items only where it does.
    static_assert(P_NUM_BARS <= 32, "a barrier per lane");
    const bool by_four = lane == P_FULL0 || lane == P_FULL1 || lane == O_FREE || lane == EPI_FULL0 || lane == EPI_FULL1 || lane >= K_STORED0;
    if constexpr (TRIO) {
      const unsigned of_item = p.store == Store::Tiles ? 7u : 6u;
      mbar_init(bar(lane), lane >= K_STORED0 ? 1u : by_four ? 4u : lane == ITEM_FREE0 || lane == ITEM_FREE1 ? of_item : 1u);
    } else {
      mbar_init(bar(lane), by_four ? 4u : lane == ITEM_FREE0 || lane == ITEM_FREE1 ? 10u : 1u);
    }
    if (lane == 0) {
      *abort_flag = 0;
      prefetch_tmap(&tmap_q);
      prefetch_tmap(&tmap_k);
      prefetch_tmap(&tmap_v);
      if (ROUTED) {
        prefetch_tmap(&tmap_key);
        prefetch_tmap(&tmap_value);
      }
    }
    mbar_fence_init();
  }
  if (!p.lengths_early) pdl_wait();
  int* seq_tiles = prefix + (MAX_BATCH + 1) - SORT_BATCH;  // for as long as the prefix sums are not there yet
  // Rank the sequences by key length, longest first (ties by index): rank = how many come before.
  if (p.batch <= SORT_BATCH) {
#pragma unroll 1
    for (int b = tid; b < p.batch; b += NTHREADS_P) {
      prefix[b] = p.cu_k[b + 1] - p.cu_k[b];  // lengths, for a moment
      seq_tiles[b] = (p.cu_q[b + 1] - p.cu_q[b] + BMT - 1) / BMT;
    }
    __syncthreads();
    int my_rank[(SORT_BATCH + NTHREADS_P - 1) / NTHREADS_P];
#pragma unroll
    for (int k = 0; k < (SORT_BATCH + NTHREADS_P - 1) / NTHREADS_P; ++k) {
      const int b = tid + k * NTHREADS_P;
      int rank = 0;
      if (b < p.batch) {
        const int mine = prefix[b];
        for (int o = 0; o < p.batch; ++o) {
          const int theirs = prefix[o];
          rank += (theirs > mine) || (theirs == mine && o < b);
        }
      }
      my_rank[k] = rank;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < (SORT_BATCH + NTHREADS_P - 1) / NTHREADS_P; ++k) {
      const int b = tid + k * NTHREADS_P;
      if (b < p.batch) order[my_rank[k]] = static_cast<unsigned short>(b);
    }
  } else {
#pragma unroll 1
    for (int b = tid; b < p.batch; b += NTHREADS_P) order[b] = static_cast<unsigned short>(b);
  }
  __syncthreads();
  if (warp == W_QK) {
    // query tiles per sequence, in that order -> exclusive prefix sum (warp scan, 32 at a time)
    int carry = 0;
#pragma unroll 1
    for (int i0 = 0; i0 < p.batch; i0 += 32) {
      const int i = i0 + lane;
      int tiles = 0;
      if (i < p.batch) {
        const int b = order[i];
        tiles = p.batch <= SORT_BATCH ? seq_tiles[b] : (p.cu_q[b + 1] - p.cu_q[b] + BMT - 1) / BMT;
      }
      int incl = tiles;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += v;
      }
      if (i < p.batch) prefix[i] = carry + incl - tiles;
      carry += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) prefix[p.batch] = carry;
  }
  if (warp == W_MMA) {
    if (TRIO) tmem_alloc(smem_u32(tmem_slot), 128, smem_u32(tmem_slot + 1), 32);
    else tmem_alloc(smem_u32(tmem_slot), TMEM_COLS);
  }
  if (p.lengths_early) pdl_wait();  // from here on q, k and v are read
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const uint32_t tmem_o = tmem + G::TMEM_O;
  auto tmem_s = [&](int st) { return TRIO ? tmem : tmem + st * 64; };                // scores of a tile
  auto tmem_p = [&](int st) { return TRIO ? tmem_slot[1] : tmem + st * 64; };  // its P

  auto read_item = [&](int it) {
    volatile int* s = slots + (it & 1) * 8;
    Item x;
    x.b = s[0]; x.h = s[1]; x.m0 = s[2]; x.q0 = s[3];
    x.Lq = s[4]; x.k0 = s[5]; x.Lk = s[6]; x.n_kv = s[7];
    return x;
  };

  // First packed row of an item's key tile j if it is one of this step's rows, to be read there; else -1.
  auto packed_row = [&](const Item& x, int j) {
    if (!ROUTED && !p.block_tables) return x.k0 + j * BN;
    const int i = j / TILES, off = x.Lk - x.Lq;
    if (!ROUTED || off < 0 || i * kBlockSize < off) return -1;
    const int row = __ldcg(p.route.tile_row + (route_first_job(x.q0, x.b) + i - (off >> 8)) * TILES + j % TILES);
    return row < 0 ? row : row & ~kRouteRagged;
  };
  // First row of any other key tile: packed too if it lies in a block that another sequence fills in this step, else in
  // the cache, through the table.
  auto cached_row = [&](const Item& x, int j, bool& packed) {
    const int i = j / TILES;
    int64_t blk = p.block_tables[x.b * p.bt_stride + i];
    if (ROUTED && i < p.max_blocks) {
      const unsigned job = __ldcg(p.route.source + x.b * p.max_blocks + i);
      if (job < static_cast<unsigned>(p.route.jobs) && __ldcg(p.route.block + job) == blk && i * kBlockSize < x.Lk - x.Lq) {
        const int row = __ldcg(p.route.tile_row + job * TILES + j % TILES);
        if (row >= 0 && !(row & kRouteRagged)) {
          packed = true;
          return row;
        }
      }
    }
    if (blk < 0 || blk >= p.num_blocks) {
      atomicOr(p.status, NVLLM_STATUS_BAD_BLOCK);
      blk = 0;
    }
    return static_cast<int>(blk * kBlockSize + (j * BN) % kBlockSize);
  };
  // A producer's record of the tiles that are stored from its stages: bit st, the tile in the stage is; bit 2 + st,
  // the parity of the stage's next completed store.  Waits for that before the stage is used again.
  auto stage_stored = [&](unsigned& stored, int st, int done) {
    if (!(stored >> st & 1u)) return true;
    const bool ok = wait_or_abort(bar(done + st), stored >> (2 + st) & 1u, abort_flag);
    stored ^= 5u << st;
    return ok;
  };
  const int64_t n_slots = p.num_blocks * kBlockSize;
  auto slot_of = [&](int64_t r) {  // of packed row r, -1: none
    const int64_t slot = p.slots[r];
    if (slot >= n_slots) atomicOr(p.status, NVLLM_STATUS_BAD_SLOT);
    return slot >= 0 && slot < n_slots ? static_cast<int>(slot) : -1;
  };

  float* inv_buf = reinterpret_cast<float*>(base_ptr + G::OFF_INV);
  // The register hand-over sits inside each group's own branch: the allocator bounds the code that
  // follows a setmaxnreg on its path, and paths that merged again would all get the smallest bound.
  if (warp >= W_QK) {
   asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(G::REGS_OTHER));
   if (warp == W_QK) {
    // ------------------------------------------------------------------ producer lane
    if (elect_one()) {
      const int hgroups = p.hq / pack;
      const int total_items = prefix[p.batch] * hgroups;
      const bool spread = (D == 128 || TRIO) && total_items > p.spread_from && (TRIO || total_items <= static_cast<int>(gridDim.x));
      int T = 0;   // key tiles loaded so far in this block's life
      unsigned stored = 0;
      // Number drawn -> item: (query tile of a sequence, head); heads vary fastest so that the blocks
      // working side by side share K/V tiles in L2.
      auto decode_item = [&](unsigned drawn) {
        Item x;
#pragma unroll 1
        while (true) {
          x.n_kv = -1;
          if (drawn >= static_cast<unsigned>(total_items)) break;
          const int idx = spread ? spread_item(drawn, prefix[p.batch], p.batch, hgroups) : static_cast<int>(drawn);
          const int pi = idx / hgroups;
          x.h = (idx - pi * hgroups) * pack;  // first of the packed heads
          int lo = 0, hi = p.batch;  // largest i with prefix[i] <= pi
#pragma unroll 1
          while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (prefix[mid] <= pi) lo = mid; else hi = mid;
          }
          x.b = order[lo];
          x.q0 = p.cu_q[x.b];
          x.Lq = p.cu_q[x.b + 1] - x.q0;
          x.k0 = p.cu_k[x.b];
          x.Lk = p.cu_k[x.b + 1] - x.k0;
          const int tiles = prefix[lo + 1] - prefix[lo];
          x.m0 = (tiles - 1 - (pi - prefix[lo])) * BMT;  // a sequence's long tiles first
          x.n_kv = key_tiles(x.m0 + BMT, x.Lq, x.Lk);
          if (x.n_kv > 0) break;
          // No visible key for the whole tile (only possible when Lk < Lq, which the engine
          // never produces): the rows are zero; written here, the other roles never see it.
#pragma unroll 1
          for (int r = x.m0; r < min(x.m0 + BMT, x.Lq); ++r) {
            uint4* dst = reinterpret_cast<uint4*>(p.out + static_cast<int64_t>(x.q0 + r) * p.out_stride + x.h * D);
#pragma unroll 1
            for (int c = 0; c < PIECES * pack; ++c) dst[c] = make_uint4(0, 0, 0, 0);  // the packed heads are adjacent
          }
          drawn = atomicAdd(&g_item_counter[counter_slot], 1u);
        }
        return x;
      };
      // The counter is read a little ahead of need -- when the loads of the current item's last
      // three key tiles are about to be issued -- so that the round trip of the atomic runs under
      // the end of the current item instead of in front of the next one.  Not earlier: an item
      // reserved long before its block is free is an item that an idle block cannot take (measured:
      // reserving at the start of the current item cost 9 % on four 4096-token sequences).
      unsigned next_draw = atomicAdd(&g_item_counter[counter_slot], 1u);
#pragma unroll 1
      for (int it = 0;; ++it) {
        const Item x = decode_item(next_draw);
        if (it >= 2 && !wait_or_abort(bar(ITEM_FREE0 + (it & 1)), ((it >> 1) - 1) & 1, abort_flag)) break;
        volatile int* s = slots + (it & 1) * 8;
        s[0] = x.b; s[1] = x.h; s[2] = x.m0; s[3] = x.q0;
        s[4] = x.Lq; s[5] = x.k0; s[6] = x.Lk; s[7] = x.n_kv;
        mbar_arrive(bar(ITEM_FULL0 + (it & 1)));
        if (x.n_kv < 0) break;

        const int kvh = x.h / p.g;
        // Q buffer: free once the last S product of the previous item is complete
        if (T > 0 && !wait_or_abort(bar(QK_DONE0 + ((T - 1) & 1)), ((T - 1) >> 1) & 1, abort_flag)) break;
        mbar_expect_tx(bar(Q_FULL), G::NSUB * pack * BMT * 128);  // the box holds pack x BMT rows per sub-tile
        tma_load_3d(base + OFF_Q, &tmap_q, bar(Q_FULL), 0, x.h, x.q0 + x.m0);
        if constexpr (G::NSUB == 2) tma_load_3d(base + OFF_Q + Q_SUB, &tmap_q, bar(Q_FULL), 64, x.h, x.q0 + x.m0);
        const int store_from = first_stored(x, p.g);
        bool ok = true;
#pragma unroll 1
        for (int j = 0; j < x.n_kv; ++j) {
          if (j == max(0, x.n_kv - 3)) next_draw = atomicAdd(&g_item_counter[counter_slot], 1u);
          const int t = T + j, st = t & 1, use = t >> 1;
          int row = packed_row(x, j);
          const bool own = row >= 0;
          bool packed = own;
          if (!own) row = cached_row(x, j, packed);
          const CUtensorMap* map = ROUTED && packed ? &tmap_key : &tmap_k;
          if (use > 0 && !(ok = wait_or_abort(bar(QK_DONE0 + st), (use - 1) & 1, abort_flag))) break;
          if (!(ok = stage_stored(stored, st, K_STORED0))) break;
          mbar_expect_tx(bar(K_FULL0 + st), KV_BYTES);
          tma_load_3d(base + OFF_K + st * KV_BYTES, map, bar(K_FULL0 + st), 0, kvh, row);
          if constexpr (G::NSUB == 2) tma_load_3d(base + OFF_K + st * KV_BYTES + KV_SUB, map, bar(K_FULL0 + st), 64, kvh, row);
          if (p.store == Store::Tiles && own && j >= store_from) {
            stored |= 1u << st;
            mbar_arrive(bar(K_DUE0 + st));
          }
        }
        if (!ok) break;
        T += x.n_kv;
      }
    }
   } else if (warp == W_V) {
    // ------------------------------------------------------------------ V producer
    // A thread of its own: a V stage is free only after the tile's P V product, and a single producer that
    // waits for that would hold back the K load of the next tile, whose stage is free much earlier.
    if (elect_one()) {
      int T = 0;
      unsigned stored = 0;
      bool ok = true;
#pragma unroll 1
      for (int it = 0; ok; ++it) {
        if (!(ok = wait_or_abort(bar(ITEM_FULL0 + (it & 1)), (it >> 1) & 1, abort_flag))) break;
        const Item x = read_item(it);
        if (x.n_kv < 0) break;
        const int kvh = x.h / p.g, store_from = first_stored(x, p.g);
#pragma unroll 1
        for (int j = 0; j < x.n_kv; ++j) {
          const int t = T + j, st = t & 1, use = t >> 1;
          int row = packed_row(x, j);
          const bool own = row >= 0;
          bool packed = own;
          if (!own) row = cached_row(x, j, packed);
          const CUtensorMap* map = ROUTED && packed ? &tmap_value : &tmap_v;
          if (use > 0 && !(ok = wait_or_abort(bar(PV_DONE0 + st), (use - 1) & 1, abort_flag))) break;
          if (!(ok = stage_stored(stored, st, V_STORED0))) break;
          mbar_expect_tx(bar(V_FULL0 + st), KV_BYTES);
          tma_load_3d(base + OFF_V + st * KV_BYTES, map, bar(V_FULL0 + st), 0, kvh, row);
          if constexpr (G::NSUB == 2) tma_load_3d(base + OFF_V + st * KV_BYTES + KV_SUB, map, bar(V_FULL0 + st), 64, kvh, row);
          if (p.store == Store::Tiles && own && j >= store_from) {
            stored |= 1u << st;
            mbar_arrive(bar(V_DUE0 + st));
          }
        }
        if (!ok) break;
        T += x.n_kv;
        mbar_arrive(bar(ITEM_FREE0 + (it & 1)));
      }
    }
   } else if (warp == W_MMA) {
    // ------------------------------------------------------------------ MMA issuer
    if (elect_one()) {
      constexpr uint32_t idesc_qk = umma_idesc(BM, BN, 0, 0);
      constexpr uint32_t idesc_pv = umma_idesc(BM, D, 0, 1);
      const uint64_t q_desc = umma_desc(base + OFF_Q, 16, 1024);
      const uint64_t k_desc = umma_desc(base + OFF_K, 16, 1024);
      const uint64_t v_desc = umma_desc(base + OFF_V, KV_SUB, 1024);
      auto issue_qk = [&](int t) -> bool {
        const int st = t & 1;
        if (!wait_or_abort(bar(K_FULL0 + st), (t >> 1) & 1, abort_flag)) return false;
        if (TRIO && t > 0 && !wait_or_abort(bar(S_FREE), (t - 1) & 1, abort_flag)) return false;
        tc_fence_after();
        const uint64_t kd = k_desc + static_cast<uint64_t>(st * (KV_BYTES >> 4));
        const uint32_t d_tmem = tmem_s(st);
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks) {
          const uint64_t qoff = ((ks >> 2) * Q_SUB + (ks & 3) * 32) >> 4;
          const uint64_t koff = ((ks >> 2) * KV_SUB + (ks & 3) * 32) >> 4;
          umma_ss(d_tmem, q_desc + qoff, kd + koff, idesc_qk, ks > 0);
        }
        umma_commit(bar(QK_DONE0 + st));
        return true;
      };
      int T = 0, nq = 0;
      bool ok = true;
#pragma unroll 1
      for (int it = 0; ok; ++it) {
        if (!(ok = wait_or_abort(bar(ITEM_FULL0 + (it & 1)), (it >> 1) & 1, abort_flag))) break;
        const Item x = read_item(it);
        if (x.n_kv < 0) break;
        if (!(ok = wait_or_abort(bar(Q_FULL), nq & 1, abort_flag))) break;
        ++nq;
#pragma unroll 1
        for (int j = -1; j < x.n_kv; ++j) {
          const int t = T + j, st = t & 1, ph = (t >> 1) & 1;
          if (j + 1 < x.n_kv && !(ok = issue_qk(t + 1))) break;  // next S runs under this tile's softmax
          if (j < 0) continue;
          if (!(ok = wait_or_abort(bar(V_FULL0 + st), ph, abort_flag))) break;
          if (!(ok = wait_or_abort(bar(P_FULL0 + st), ph, abort_flag))) break;
          // the first product of an item overwrites O: the previous item's O must have been read (two groups: by the warps
          // that have just filled P)
          if (!TRIO && j == 0 && it > 0 && !(ok = wait_or_abort(bar(O_FREE), (it - 1) & 1, abort_flag))) break;
          tc_fence_after();
          const uint64_t vd = v_desc + static_cast<uint64_t>(st * (KV_BYTES >> 4));
          const uint32_t p_tmem = tmem_p(st);
#pragma unroll
          for (int ks = 0; ks < BN / 16; ++ks)
            umma_ts(tmem_o, p_tmem + ks * 8, vd + static_cast<uint64_t>((ks * 2048) >> 4), idesc_pv,
                    (j > 0 || ks > 0) ? 1u : 0u);
          umma_commit(bar(PV_DONE0 + st));
        }
        if (!ok) break;
        T += x.n_kv;
        mbar_arrive(bar(ITEM_FREE0 + (it & 1)));
      }
      if (!ok) {  // make sure nothing is still running on TMEM before it is freed
        umma_commit(bar(DRAIN));
        (void)mbar_wait(bar(DRAIN), 0);
      }
    }
   } else if (p.store != Store::None && (TRIO || !ROUTED)) {
    // -------------------------------------------------- a warp left: packed rows to the cache
    if constexpr (TRIO) {
      // Those of key tiles, which the epilogue warps store where there are any: the same, by one warp.
      constexpr int ROWS = 32 / PIECES;
      const int piece = lane % PIECES;
      const int64_t row_elems = static_cast<int64_t>(p.hkv) * D;
      int T = 0;
      unsigned due = 0;  // bit st: parity of stage st's next K_DUE and V_DUE
      bool ok = p.store == Store::Tiles;
#pragma unroll 1
      for (int it = 0; ok; ++it) {
        if (!(ok = wait_or_abort(bar(ITEM_FULL0 + (it & 1)), (it >> 1) & 1, abort_flag))) break;
        const Item x = read_item(it);
        if (x.n_kv < 0) break;
        const int64_t col = static_cast<int64_t>(x.h / p.g) * D + piece * 8;
#pragma unroll 1
        for (int j = first_stored(x, p.g); ok && j < x.n_kv; ++j) {
          const int t = T + j, st = t & 1;
          const int64_t row0 = packed_row(x, j);
          if (row0 < 0) continue;  // read through the table: stored already
          const int n_rows = static_cast<int>(min(static_cast<int64_t>(min(BN, x.Lk - j * BN)), p.n_new - row0));
          int slot[2];  // of rows lane and 32 + lane
#pragma unroll
          for (int i = 0; i < 2; ++i) slot[i] = i * 32 + lane < n_rows ? slot_of(row0 + i * 32 + lane) : -1;
#pragma unroll 1
          for (int kv = 0; kv < 2; ++kv) {
            if (!(ok = wait_or_abort(bar((kv ? V_DUE0 : K_DUE0) + st), due >> st & 1, abort_flag))) break;
            if (!(ok = wait_or_abort(bar((kv ? V_FULL0 : K_FULL0) + st), (t >> 1) & 1, abort_flag))) break;
            const uint32_t src = base + (kv ? OFF_V : OFF_K) + st * KV_BYTES + (piece >> 3) * KV_SUB;
            __nv_bfloat16* cache = (kv ? p.v_store : p.k_store) + col;
#pragma unroll 1
            for (int r0 = 0; r0 < BN; r0 += 16) {
              uint4 v[16 / ROWS];
#pragma unroll
              for (int i = 0; i < 16 / ROWS; ++i) {
                const int r = r0 + i * ROWS + lane / PIECES;
                v[i] = ld_shared16(src + r * 128 + (((piece ^ r) & 7) << 4));
              }
#pragma unroll
              for (int i = 0; i < 16 / ROWS; ++i) {
                const int to = __shfl_sync(0xffffffffu, r0 < 32 ? slot[0] : slot[1], r0 % 32 + i * ROWS + lane / PIECES);
                if (to >= 0) *reinterpret_cast<uint4*>(cache + to * row_elems) = v[i];
              }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(bar((kv ? V_STORED0 : K_STORED0) + st));
          }
          due ^= 1u << st;
        }
        T += x.n_kv;
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(ITEM_FREE0 + (it & 1)));
      }
    }
    // All of them, or those that no item has a tile of: of sequences without a query row, in front of the first
    // sequence and behind the last.  A 16-byte piece of a K and a V row per lane, two such at a time.
    const uint32_t per_row = p.hkv * PIECES;
    const bool all = p.store == Store::Spare;
    int b = ROUTED ? p.batch + 1 : all ? p.batch : static_cast<int>(blockIdx.x) - static_cast<int>(gridDim.x);
#pragma unroll 1
    while (b <= p.batch) {
      int64_t from = 0, to = p.n_new;
      uint32_t first = blockIdx.x, step = gridDim.x;
      if (all || b == p.batch) {
        if (!all) from = p.cu_k[p.batch];
        b = p.batch + 1;
      } else if (b < 0) {
        to = p.cu_k[0];
        b += gridDim.x;
        b = min(b, p.batch);
      } else {
        from = p.cu_k[b], to = p.cu_q[b + 1] == p.cu_q[b] ? p.cu_k[b + 1] : from;
        first = 0, step = 1;
        b = min(b + static_cast<int>(gridDim.x), p.batch);
      }
      const uint32_t total = static_cast<uint32_t>(max(min(to, p.n_new) - from, static_cast<int64_t>(0)) * per_row);
#pragma unroll 1
      for (uint32_t i0 = first * 32 + lane; i0 < total; i0 += 2 * step * 32) {
        uint4 kreg[2], vreg[2];
        int64_t dst[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const uint32_t i = i0 + u * step * 32, row = i / per_row, piece = i - row * per_row;
          dst[u] = -1;
          if (i >= total) continue;
          const int slot = slot_of(from + row);
          if (slot >= 0) dst[u] = static_cast<int64_t>(slot) * per_row + piece;
          kreg[u] = __ldg(reinterpret_cast<const uint4*>(p.k + (from + row) * p.k_stride) + piece);
          vreg[u] = __ldg(reinterpret_cast<const uint4*>(p.v + (from + row) * p.v_stride) + piece);
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          if (dst[u] < 0) continue;
          reinterpret_cast<uint4*>(p.k_store)[dst[u]] = kreg[u];
          reinterpret_cast<uint4*>(p.v_store)[dst[u]] = vreg[u];
        }
      }
    }
   }
  } else if (warp < 4) {
    // ------------------------------------------------------------------ softmax rows
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(G::REGS_SOFTMAX));
    const int r = warp * 32 + lane;
    const int r_tok = token_of(r);  // this row's token within the tile (== BMT for the unused rows of a 7-head tile)
    const uint32_t lane_addr = static_cast<uint32_t>(warp * 32) << 16;
    int T = 0;
    bool ok = true;
#pragma unroll 1
    for (int it = 0; ok; ++it) {
      if (!(ok = wait_or_abort(bar(ITEM_FULL0 + (it & 1)), (it >> 1) & 1, abort_flag))) break;
      const Item x = read_item(it);
      if (x.n_kv < 0) break;
      const int qi = x.m0 + r_tok, off = x.Lk - x.Lq;
      float m_used = -INFINITY, l = 0.f;
#pragma unroll 1
      for (int j = 0; j < x.n_kv; ++j) {
        const int t = T + j, st = t & 1, ph = (t >> 1) & 1;
        const uint32_t scores = tmem_s(st) + lane_addr;
        if (!(ok = wait_or_abort(bar(QK_DONE0 + st), ph, abort_flag))) break;
        tc_fence_after();
        uint32_t s[64];
        tmem_ld32(scores, *reinterpret_cast<uint32_t(*)[32]>(&s[0]));
        tmem_ld32(scores + 32, *reinterpret_cast<uint32_t(*)[32]>(&s[32]));
        tmem_wait_ld();
        if (TRIO) {  // the next tile's scores may be written
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(bar(S_FREE));
        }

        const int j0 = j * BN;
        if ((j0 + BN - 1 > x.m0 + off) || (j0 + BN > x.Lk)) {  // tile touches the diagonal or the end
          const int limit = min(qi + off, x.Lk - 1) - j0;        // columns c <= limit are visible
#pragma unroll
          for (int c = 0; c < 64; ++c)
            if (c > limit) s[c] = 0xff800000u;  // -inf
        }
        float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int c = 0; c < 64; c += 8) {
          mx4[0] = fmax3(mx4[0], __uint_as_float(s[c]), __uint_as_float(s[c + 1]));
          mx4[1] = fmax3(mx4[1], __uint_as_float(s[c + 2]), __uint_as_float(s[c + 3]));
          mx4[2] = fmax3(mx4[2], __uint_as_float(s[c + 4]), __uint_as_float(s[c + 5]));
          mx4[3] = fmax3(mx4[3], __uint_as_float(s[c + 6]), __uint_as_float(s[c + 7]));
        }
        const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
        const float m_new = fmaxf(m_used, mx * p.scale_log2e);
        // lazy rescale: keep the old reference maximum unless it has been outgrown by 2^8
        const bool grow = m_new > m_used + kRescaleThreshold;
        if (__any_sync(0xffffffffu, grow)) {
          float alpha = 1.f;
          if (grow) {
            alpha = (m_used == -INFINITY) ? 0.f : fast_exp2(m_used - m_new);
            m_used = m_new;
            l *= alpha;
          }
          if (j > 0) {  // O holds tiles 0..j-1 of this item once the previous P V product has finished
            if (!(ok = wait_or_abort(bar(PV_DONE0 + ((t - 1) & 1)), ((t - 1) >> 1) & 1, abort_flag))) break;
            tc_fence_after();
#pragma unroll 1
            for (int c = 0; c < OCH; ++c) {
              uint32_t o[32];
              tmem_ld32(tmem_o + lane_addr + c * 32, o);
              tmem_wait_ld();
#pragma unroll
              for (int e = 0; e < 32; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * alpha);
              tmem_st32(tmem_o + lane_addr + c * 32, o);
            }
          }
        }
        const float msub = (m_used == -INFINITY) ? 0.f : m_used;
        // p = 2^(s * scale - m): the multiply-subtract and the row sum run two lanes at a time
        const uint64_t scale2 = pack2(p.scale_log2e, p.scale_log2e), nmsub2 = pack2(-msub, -msub);
        uint64_t sum2[2] = {0ull, 0ull};
#pragma unroll
        for (int c = 0; c < 32; ++c) {  // P is packed in place: s[c] <- (p[2c], p[2c+1])
          float a0, a1;
          unpack2(fma2(pack2(__uint_as_float(s[2 * c]), __uint_as_float(s[2 * c + 1])), scale2, nmsub2), a0, a1);
          const float p0 = fast_exp2(a0), p1 = fast_exp2(a1);
          sum2[c & 1] = add2(sum2[c & 1], pack2(p0, p1));
          s[c] = pack_bf16x2(p0, p1);
        }
        {
          float t0, t1, t2, t3;
          unpack2(sum2[0], t0, t1);
          unpack2(sum2[1], t2, t3);
          l += (t0 + t1) + (t2 + t3);
        }
        if (j0 + BN > x.Lk) {
          // Last tile of the sequence: V rows past the end hold whatever the cache block (or the
          // next sequence) has there.  Their P is 0, but 0 x NaN would still poison O, so the
          // rows are cleared in shared memory before the product is issued.
          if (!(ok = wait_or_abort(bar(V_FULL0 + st), ph, abort_flag))) break;
          const int first = x.Lk - j0;  // rows [first, 64) are dead
          unsigned char* vt = base_ptr + OFF_V + st * KV_BYTES;
#pragma unroll 1
          for (int i = r; i < (BN - first) * PIECES; i += 128) {
            const int row = first + i / PIECES, piece = i % PIECES;
            *reinterpret_cast<uint4*>(vt + (piece >> 3) * KV_SUB + row * 128 + (piece & 7) * 16) = make_uint4(0, 0, 0, 0);
          }
          fence_proxy_async();
        }
        if (TRIO && j > 0) {  // P has one place: the product of the tile before must have read it
          if (!(ok = wait_or_abort(bar(PV_DONE0 + ((t - 1) & 1)), ((t - 1) >> 1) & 1, abort_flag))) break;
          tc_fence_after();
        }
        tmem_st32(TRIO ? tmem_p(st) + lane_addr : scores, *reinterpret_cast<uint32_t(*)[32]>(&s[0]));
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(P_FULL0 + st));
      }
      if (!ok) break;
      T += x.n_kv;

      const float inv = l > 0.f ? 1.f / l : 0.f;
      if constexpr (TRIO) {
        if (!(ok = wait_or_abort(bar(PV_DONE0 + ((T - 1) & 1)), ((T - 1) >> 1) & 1, abort_flag))) break;
        tc_fence_after();
        // O / l -> bf16, 32 columns at a time through this warp's patch of shared memory, as an epilogue warp does it
        unsigned char* stage = base_ptr + G::OFF_STAGE + warp * 2048;
        const int srow = lane >> 2, spiece = lane & 3;
        __nv_bfloat16* out_tile = p.out + static_cast<int64_t>(x.q0 + x.m0) * p.out_stride + x.h * D;
        const int toks_valid = min(BMT, x.Lq - x.m0);
#pragma unroll (ROUTED ? 1 : OCH)
        for (int c = 0; c < OCH; ++c) {
          uint32_t o[32];
          tmem_ld32(tmem_o + lane_addr + c * 32, o);
          tmem_wait_ld();
          uint4 v[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            v[k].x = pack_bf16x2(__uint_as_float(o[8 * k]) * inv, __uint_as_float(o[8 * k + 1]) * inv);
            v[k].y = pack_bf16x2(__uint_as_float(o[8 * k + 2]) * inv, __uint_as_float(o[8 * k + 3]) * inv);
            v[k].z = pack_bf16x2(__uint_as_float(o[8 * k + 4]) * inv, __uint_as_float(o[8 * k + 5]) * inv);
            v[k].w = pack_bf16x2(__uint_as_float(o[8 * k + 6]) * inv, __uint_as_float(o[8 * k + 7]) * inv);
          }
#pragma unroll
          for (int k = 0; k < 4; ++k) *reinterpret_cast<uint4*>(stage + lane * 64 + ((k ^ ((lane >> 1) & 3)) << 4)) = v[k];
          __syncwarp();
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int lr = i * 8 + srow, row = warp * 32 + lr;  // of the warp's 32, of the tile
            const int tok = token_of(row), hh = row - tok * pack;
            const uint4 v = *reinterpret_cast<const uint4*>(stage + lr * 64 + ((spiece ^ ((lr >> 1) & 3)) << 4));
            if (tok < toks_valid)
              *reinterpret_cast<uint4*>(out_tile + static_cast<int64_t>(tok) * p.out_stride + hh * D + c * 32 + spiece * 8) = v;
          }
          __syncwarp();
        }
        tc_fence_before();
        if (lane == 0) mbar_arrive(bar(ITEM_FREE0 + (it & 1)));
      } else {
        // the row's normaliser goes to the epilogue warps; this warp is done with the item
        inv_buf[(it & 1) * 128 + r] = inv;
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(bar(EPI_FULL0 + (it & 1)));
          mbar_arrive(bar(ITEM_FREE0 + (it & 1)));
        }
      }
    }
  } else if constexpr (!TRIO) {
    // ------------------------------------------------------------------ epilogue rows
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(G::REGS_EPILOGUE));
    // Same rows as softmax warp (warp - 4): a warp reaches the TMEM lanes 32 x (warp mod 4).
    const int ew = warp - 4, r = ew * 32 + lane;
    const uint32_t lane_addr = static_cast<uint32_t>(ew * 32) << 16;
    unsigned char* stage = base_ptr + G::OFF_STAGE + ew * 2048;  // this warp's 32 rows x 64 B
    int T = 0;
    unsigned due = 0;  // bit st: parity of stage st's next K_DUE and V_DUE
    bool ok = true;
#pragma unroll 1
    for (int it = 0; ok; ++it) {
      if (!(ok = wait_or_abort(bar(ITEM_FULL0 + (it & 1)), (it >> 1) & 1, abort_flag))) break;
      const Item x = read_item(it);
      if (x.n_kv < 0) break;
      if (p.store == Store::Tiles) {
        // Packed rows to the cache: the first item of a sequence that loads a key tile writes its rows to their slots
        // from shared memory, 16 of the 64 per warp, 512 bytes with an instruction.
        constexpr int ROWS = 32 / PIECES;  // rows that a warp writes at a time
        const int piece = lane % PIECES;
        const int64_t row_elems = static_cast<int64_t>(p.hkv) * D;
        const int64_t col = static_cast<int64_t>(x.h / p.g) * D + piece * 8;
#pragma unroll 1
        for (int j = first_stored(x, p.g); j < x.n_kv; ++j) {
          const int t = T + j, st = t & 1, r_warp = ew * 16;
          const int64_t row0 = packed_row(x, j);
          if (row0 < 0) continue;  // read through the table: stored already
          const int64_t n_rows = min(static_cast<int64_t>(min(BN, x.Lk - j * BN)), p.n_new - row0);
          const int slot = lane < 16 && r_warp + lane < n_rows ? slot_of(row0 + r_warp + lane) : -1;
          // A stage's barrier tells its phase by parity only, and these warps do not wait for every tile: between
          // the producer's word that the load is issued and theirs that it is stored it stays at this tile's.
#pragma unroll 1
          for (int kv = 0; ok && kv < 2; ++kv) {
            if (!(ok = wait_or_abort(bar((kv ? V_DUE0 : K_DUE0) + st), due >> st & 1, abort_flag))) break;
            if (!(ok = wait_or_abort(bar((kv ? V_FULL0 : K_FULL0) + st), (t >> 1) & 1, abort_flag))) break;
            const uint32_t src = base + (kv ? OFF_V : OFF_K) + st * KV_BYTES + (piece >> 3) * KV_SUB + r_warp * 128;
            __nv_bfloat16* cache = (kv ? p.v_store : p.k_store) + col;
            uint4 v[16 / ROWS];
#pragma unroll
            for (int i = 0; i < 16 / ROWS; ++i) {  // all in flight before the first is written: one after the other took 1700 cycles
              const int r = i * ROWS + lane / PIECES;
              v[i] = ld_shared16(src + r * 128 + (((piece ^ r) & 7) << 4));
            }
#pragma unroll
            for (int i = 0; i < 16 / ROWS; ++i) {
              const int to = __shfl_sync(0xffffffffu, slot, i * ROWS + lane / PIECES);
              if (to >= 0) *reinterpret_cast<uint4*>(cache + to * row_elems) = v[i];
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(bar((kv ? V_STORED0 : K_STORED0) + st));
          }
          if (!ok) break;
          due ^= 1u << st;
        }
        if (!ok) break;
      }
      T += x.n_kv;
      if (!(ok = wait_or_abort(bar(EPI_FULL0 + (it & 1)), (it >> 1) & 1, abort_flag))) break;
      const float inv = inv_buf[(it & 1) * 128 + r];
      // epilogue: O / l -> bf16; 32 columns at a time through this warp's patch of shared memory
      if (!(ok = wait_or_abort(bar(PV_DONE0 + ((T - 1) & 1)), ((T - 1) >> 1) & 1, abort_flag))) break;
      tc_fence_after();
      // lane -> (row, 16-byte piece) of the eight 64-byte row segments one store instruction writes
      const int srow = lane >> 2, spiece = lane & 3;
      __nv_bfloat16* out_tile = p.out + static_cast<int64_t>(x.q0 + x.m0) * p.out_stride + x.h * D;
      const int toks_valid = min(BMT, x.Lq - x.m0);
      // unrolled where a block has few items (a prompt of 201 tokens 9.0 us, 9.1 rolled up); through the route tables it
      // has many, and the instructions count (64 prompts 121 -> 118.6)
#pragma unroll (ROUTED ? 1 : 4)
      for (int c = 0; c < OCH; ++c) {
        uint32_t o[32];
        tmem_ld32(tmem_o + lane_addr + c * 32, o);
        tmem_wait_ld();
        if (c == OCH - 1) {  // O is in registers: the next item's first product may overwrite it
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(bar(O_FREE));
        }
        uint4 v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          v[k].x = pack_bf16x2(__uint_as_float(o[8 * k]) * inv, __uint_as_float(o[8 * k + 1]) * inv);
          v[k].y = pack_bf16x2(__uint_as_float(o[8 * k + 2]) * inv, __uint_as_float(o[8 * k + 3]) * inv);
          v[k].z = pack_bf16x2(__uint_as_float(o[8 * k + 4]) * inv, __uint_as_float(o[8 * k + 5]) * inv);
          v[k].w = pack_bf16x2(__uint_as_float(o[8 * k + 6]) * inv, __uint_as_float(o[8 * k + 7]) * inv);
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) *reinterpret_cast<uint4*>(stage + lane * 64 + ((k ^ ((lane >> 1) & 3)) << 4)) = v[k];
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int lr = i * 8 + srow;       // row within the warp's 32
          const int row = ew * 32 + lr;      // row of the tile
          const int tok = token_of(row), hh = row - tok * pack;
          const uint4 v = *reinterpret_cast<const uint4*>(stage + lr * 64 + ((spiece ^ ((lr >> 1) & 3)) << 4));
          if (tok < toks_valid)
            *reinterpret_cast<uint4*>(out_tile + static_cast<int64_t>(tok) * p.out_stride + hh * D + c * 32 + spiece * 8) = v;
        }
        __syncwarp();
      }
      if (lane == 0) mbar_arrive(bar(ITEM_FREE0 + (it & 1)));
    }
  }

  tc_fence_before();
  __syncthreads();
  if (tid == 0) {
    if (*abort_flag) atomicOr(p.status, NVLLM_STATUS_TIMEOUT);
    // the last block to leave re-arms this launch slot's counters
    if (atomicAdd(&g_done_counter[counter_slot], 1u) == gridDim.x - 1) {
      g_item_counter[counter_slot] = 0;
      g_done_counter[counter_slot] = 0;
      __threadfence();
    }
  }
  if (warp == W_MMA) {
    tc_fence_after();
    tmem_dealloc(tmem, TRIO ? 128 : TMEM_COLS);
    if (TRIO) tmem_dealloc(tmem_slot[1], 32);
  }
}

// ---- host side ---------------------------------------------------------------------------

static std::atomic<unsigned> g_launch_seq{0};  // its launches take the counter slots in turn, whatever their kernel

// Heads packed into a query tile: the largest divisor of the group size that is at most 8
// (NVLLM_PREFILL_PACK = 1..8 caps it; measurement aid, read on every call).
static int heads_per_tile(int g) {
  int cap = 8, pack = 1;
  if (const char* s = std::getenv("NVLLM_PREFILL_PACK")) cap = std::atoi(s);
  for (int n = 2; n <= 8 && n <= cap; ++n)
    if (g % n == 0) pack = n;
  return pack;
}

static int64_t max_items_of(int hq, int pack, int max_seqlen_q, int batch) {
  const int bmt = tc::BM / pack;
  return static_cast<int64_t>((max_seqlen_q + bmt - 1) / bmt) * (hq / pack) * batch;
}

int64_t prefill_max_items(int hq, int hkv, int max_seqlen_q, int batch) {
  return max_items_of(hq, heads_per_tile(hq / hkv), max_seqlen_q, batch);
}

// Prompts of less than four key tiles are the two-block form's: a block of three has no warps to write an item's results while
// the next is begun (24 prompts of 192 tokens, 14 / 2 heads, two blocks -> three 14.1 -> 15.0 us, 100 of 100-200 26.9 -> 27.4; of 256 20.7 -> 19.8).
constexpr int kTrioTokens = 4 * tc::BN;

// All prompts have the same number of query tiles, as far as their sum and the longest tell (through a table, where one prompt with
// a cached block may take all that is missing, for sure; else if they are spread evenly up to the longest): in launches of three
// blocks to an SM their long tiles go first.  Sequence after sequence the last ones' start late and run alone at the end.  Three
// blocks, 14 / 2 heads, without -> with that order, us: 4 of 4096 tokens 189 -> 166, 16 of 1024 62.4 -> 56.2, 8 of 512 19.8 -> 15.9.
// Where a prompt has a tile more than others the turns do not line up (two blocks -> three with the order: 6 of 500-510 tokens, 28
// or 29 tiles, 15.1 -> 18.3, 12 of 250-255 12.8 -> 14.4; 16 / 16 heads, 5 of 2048 of which one has a cached block 80.4 -> 96.1).  Not with two
// blocks, whose short launches the code for it costs 1-1.7 %, nor at head_dim 128 (4 of 4096 242 -> 247, 64 of 256 50 -> 61: what
// keeps memory busy there is the mix of long and short tiles).
static bool same_tiles(const PrefillParams& p, int64_t total_q, int bmt) {
  const int64_t missing = static_cast<int64_t>(p.max_seqlen_q) * p.batch - total_q;  // to prompts that are all as long as the longest
  const int in_last = (p.max_seqlen_q - 1) % bmt + 1;                               // tokens of that one's last tile
  return p.batch > 1 && (p.block_tables ? missing < in_last : 2 * missing < static_cast<int64_t>(in_last) * p.batch);
}

// Head_dim 64: three blocks to an SM, of eight warps, or two of twelve.  Three get up to 20 % more done where there is enough
// for all of them, since an item takes a block of three longer.
// Prompts of the same number of tiles: more than two items to an SM, and eight query tiles to a prompt, since the rows of a key
// tile are stored by one warp instead of four, the oftener the fewer query tiles read it.  Two blocks -> three, us: 4 of 4096
// tokens, 14 / 2 heads 180 -> 165, 16 of 1024 62.9 -> 56.2, 4 of 1024 24.8 -> 21.4, 10 of 300 13.3 -> 13.1; 7 / 1 heads, 5 of 2048 46.6 -> 35.6;
// 32 / 8, 8 of 512 27.3 -> 25.3; 16 / 16, 8 of 2048 123 -> 111.  On the other side 16 / 16 heads, 48 of 256 (two tiles) 34.9 -> 42.9, 32 of 512
// (four) 52.4 -> 58.3.
// Other prompts, several heads to a tile: eight times the longest item's key tiles for every SM, or four times from twelve
// prompts of different lengths on: 64 of 100-1024 tokens, 14 / 2 heads, 73.9 -> 71.2, 48 of 200-800 63.1 -> 60.6.  On the other side 5 of
// 2000-4096 (4.4 times) 108 -> 114, 16 of 1000-1024 (6.4 times) 62.7 -> 66.1; one head to a tile, 48 of 200-400 (8 times) 46.8 -> 51.3.
// Of 237 launches that the rule takes (six pairs of heads, 256 to 4096 tokens) the mean is 6 % faster; 21 are slower, six of them
// by 3-8 % (32 / 8 heads, 7 of 256 13.1 -> 14.1; 16 / 16, 3 of 1024 22.0 -> 23.0).
static bool three_blocks(const PrefillParams& p, int64_t total_q, int sms, int pack) {
  const int bmt = tc::BM / pack;
  const double mean = static_cast<double>(total_q) / p.batch;
  const double items = static_cast<double>(total_q) / bmt * (p.hq / pack), tiles = items * (mean / 2 + tc::BN / 2) / tc::BN;
  if (mean < kTrioTokens) return false;
  if (same_tiles(p, total_q, bmt)) return mean > 7 * bmt && items > 2.0 * sms;
  const double times = tiles * tc::BN / (static_cast<double>(sms) * p.max_seqlen_k);
  return pack > 1 && (times >= 8 || (times >= 4 && p.batch >= 12 && p.max_seqlen_q >= 1.03 * mean));
}

PrefillPlan prefill_plan(const PrefillParams& p, int64_t total_q, int sms) {
  PrefillPlan plan;
  plan.pack = heads_per_tile(p.g);  // reads the environment: once to a launch
  const int bmt = tc::BM / plan.pack;
  const bool routed = p.route.jobs > 0;
  plan.blocks = p.d == 64 && three_blocks(p, total_q, sms, plan.pack) ? 3 : 2;
  // an upper bound of the work items known to the host: no more blocks than that
  const int64_t max_items = max_items_of(p.hq, plan.pack, p.max_seqlen_q, p.batch);
  plan.grid = plan.blocks * sms;
  // With an item to a block and more items than SMs, blocks that share an SM with those of long tiles get short ones by
  // another order: 6 prompts of 300 tokens 15.1 -> 13.4 us, 10 of 100 11.4 -> 10.4, 3 of 500 14.6 -> 14.1.  Which blocks
  // meet on an SM is the hardware's choice, so this is a matter of averages: of 448 launches of 2-40 prompts (eight
  // pairs of head counts) the 346 that the rule takes are 6 % faster in the mean, twelve of them 1-10 % slower (22 of
  // 381-420 tokens, 2 / 1 heads, 12.9 -> 14.4).  Not where an SM has one block (the divisions cost 0.3 us: 5 prompts of 60
  // tokens 8.2 -> 8.5), where long and short prompts mix, whose tiles every q-th of the list does not line up (19 of
  // 209-582 16.0 -> 17.3), nor at head_dim 64 (14 / 2 heads, 6 of 100-300 tokens 9.65 -> 10.05).
  const bool alike = p.max_seqlen_q <= 5 * bmt || 20ll * p.max_seqlen_q * p.batch <= 23 * total_q;
  plan.spread_from = plan.blocks == 3 ? (same_tiles(p, total_q, bmt) ? 0 : 1 << 30) : p.d == 128 && p.batch > 1 && alike ? sms : 1 << 30;
  // Rows to be stored.  Where blocks work on several items one after the other, from the key tiles that pass through
  // shared memory (64 prompts of 100-1024 tokens, 16 / 8 heads: 200 us when two idle warps of every block copied all
  // rows, 4 KB in flight; 120 from the tiles; 110 with nothing to store).  Where a block has one item at most that
  // would end it later (a prompt of 201 tokens 9.05 -> 9.5 us): there an idle warp of every block copies the rows, by
  // as many blocks as that takes two trips of, as long as four of them are enough (6 prompts of 300 tokens: 15.8
  // us from the tiles, 20.2 copied).
  const int64_t pieces = p.n_new * p.hkv * (p.d / 8);
  plan.store = !p.slots ? Store::None : routed || max_items > plan.grid || pieces > 4ll * 64 * plan.grid ? Store::Tiles : Store::Spare;
  const int64_t copy_blocks = plan.store == Store::Spare ? (pieces + 127) / 128 : 0;
  plan.grid = static_cast<int>(std::min<int64_t>(plan.grid, std::max(max_items, copy_blocks)));
  return plan;
}

// Makes the kernels of a form ready for their launches on a device.
template <int D, bool TRIO>
static int prepare_prefill_tcp() {
  for (auto kernel : {prefill_tcp_kernel<D, false, TRIO>, prefill_tcp_kernel<D, true, TRIO>}) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, tcp::Geo<D, TRIO>::SMEM);
    if (e != cudaSuccess) return fail(NVLLM_E_CUDA, "prefill (persistent): set-up failed: %s", cudaGetErrorString(e));
    // The warp groups trade registers inside the pool the block gets at launch (threads x the kernel's
    // register count); a build whose count is below the assumed 80 could never satisfy the softmax
    // group's request, and that request waits without a bound.
    cudaFuncAttributes attr;
    e = cudaFuncGetAttributes(&attr, kernel);
    if (e != cudaSuccess) return fail(NVLLM_E_CUDA, "prefill (persistent): set-up failed: %s", cudaGetErrorString(e));
    if (attr.numRegs < tcp::REGS_LAUNCH)
      return fail(NVLLM_E_CUDA, "prefill (persistent): built with %d registers per thread, the warp groups' hand-over needs %d",
                  attr.numRegs, tcp::REGS_LAUNCH);
  }
  return NVLLM_OK;
}

template <int D, bool TRIO>
static int launch_prefill_tcp_t(const PrefillParams& p_in, const PrefillPlan& plan, int64_t total_q, int64_t total_k, cudaStream_t stream) {
  using G = tcp::Geo<D, TRIO>;
  static bool ready[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return fail(NVLLM_E_NO_DEVICE, "prefill: device index %d out of range", dev);
  if (p_in.out_stride > (1 << 23)) return fail(NVLLM_E_GEOMETRY, "prefill: out row stride %lld too large", (long long)p_in.out_stride);
  if (!ready[dev]) {  // all forms of this head_dim: another's first launch may be captured
    int rc = prepare_prefill_tcp<D, false>();
    if (D == 64 && rc == NVLLM_OK) rc = prepare_prefill_tcp<64, true>();
    if (rc) return rc;
    ready[dev] = true;
  }
  PrefillParams p = p_in;
  const bool routed = p.route.jobs > 0;
  p.pack = plan.pack;
  const int pack = p.pack, bmt = tc::BM / pack;
  p.tile_tokens = bmt;
  p.inv_pack = 65536 / pack + 1;  // exact for rows of a tile
  CUtensorMap mq, mk, mv, mkey, mvalue;
  if (!make_tmap_3d(&mq, p.q, D, p.hq, total_q, D, p.q_stride, bmt, pack)) return NVLLM_E_CUDA;
  if (p.block_tables) {
    const uint64_t slots = static_cast<uint64_t>(p.num_blocks) * kBlockSize;
    const uint64_t row = static_cast<uint64_t>(p.hkv) * D;
    if (!make_tmap_3d(&mk, p.k, D, p.hkv, slots, D, row, tc::BN)) return NVLLM_E_CUDA;
    if (!make_tmap_3d(&mv, p.v, D, p.hkv, slots, D, row, tc::BN)) return NVLLM_E_CUDA;
    if (routed) {
      if (!make_tmap_3d(&mkey, p.key, D, p.hkv, p.n_new, D, p.key_stride, tc::BN)) return NVLLM_E_CUDA;
      if (!make_tmap_3d(&mvalue, p.value, D, p.hkv, p.n_new, D, p.value_stride, tc::BN)) return NVLLM_E_CUDA;
    } else {
      mkey = mk, mvalue = mv;
    }
  } else {
    if (!make_tmap_3d(&mk, p.k, D, p.hkv, total_k, D, p.k_stride, tc::BN)) return NVLLM_E_CUDA;
    if (!make_tmap_3d(&mv, p.v, D, p.hkv, total_k, D, p.v_stride, tc::BN)) return NVLLM_E_CUDA;
    mkey = mk, mvalue = mv;
  }
  p.spread_from = plan.spread_from;
  p.store = plan.store;
  static_assert(sizeof(g_launch_seq) == 4 && (1ull << 32) % tcp::NUM_SLOTS == 0, "the slots follow one another when the count wraps");
  const int slot = static_cast<int>(g_launch_seq.fetch_add(1) % tcp::NUM_SLOTS);
  return launch_kernel("prefill (tcgen05, persistent)", routed ? prefill_tcp_kernel<D, true, TRIO> : prefill_tcp_kernel<D, false, TRIO>, dim3(plan.grid),
                       dim3(G::NTHREADS), G::SMEM, stream, p, mq, mk, mv, mkey, mvalue, slot);
}

int launch_prefill_tcp(const PrefillParams& p, int64_t total_q, int64_t total_k, cudaStream_t stream) {
  const int sms = num_sms();
  if (sms <= 0) return fail(NVLLM_E_NO_DEVICE, "prefill: no CUDA device is usable");
  const PrefillPlan plan = prefill_plan(p, total_q, sms);
  if (p.d == 128) return launch_prefill_tcp_t<128, false>(p, plan, total_q, total_k, stream);
  return plan.blocks == 3 ? launch_prefill_tcp_t<64, true>(p, plan, total_q, total_k, stream)
                          : launch_prefill_tcp_t<64, false>(p, plan, total_q, total_k, stream);
}

}  // namespace nvllm
