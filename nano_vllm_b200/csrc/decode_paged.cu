// Paged GQA decode attention (one query token per sequence) for sm_100a.
//
// Math follows the decode branch of nanovllm/layers/attention.py:74-77
// (flash_attn_with_kvcache over a block table): out[b,h] = softmax(scale q.K^T) V over the
// first context_lens[b] cached tokens, query head h reading KV head h / G.  The step variant
// also does what store_kvcache does just before it (attention.py:65-66) for the one new token
// of every sequence.
//
// Design (HBM-bandwidth bound; every cached byte is read exactly once, by a fixed set of
// resident thread blocks that all finish together):
//   * The batch is cut into work units of UNIT = NW x TT tokens (64 for head_dim 128).  The
//     units of all sequences, in batch order, form one list; it is split into `n_ranges` equal
//     contiguous ranges, and thread block (range s, KV head g) streams range s of KV head g.
//     The grid is n_ranges x Hkv = two blocks per SM, a function of host-visible sizes only, so
//     the launch can be captured in a CUDA graph.  Every block derives the split from
//     context_lens itself (a block-wide scan of the units per sequence), so blocks carry the
//     same number of bytes whatever the lengths are: no tail of half-empty waves, one ramp-up.
//   * Warp w of a thread block owns the TT-token tile w of every unit and runs its own NST-stage
//     cp.async ring (16-byte copies, XOR-swizzled rows so ldmatrix is conflict free).  The ring keeps
//     running across sequence boundaries.  Rows past the end of a context are zero-filled, never read.
//     The Plain variant has the warps meet at every unit, so that a block's reads stay within a stretch
//     of memory instead of spreading over as many as it has warps: 256 sequences of 2048-8192 tokens
//     (32 / 8 heads) 731 -> 717 us in a chain, 805 -> 777 alone behind a flush of L2, one of 8 ranks' shard
//     of it 133 -> 127, 48 of 32768 (head_dim 64, layer) 126.3 -> 122.7, 512 of 100-1024 (16 / 8 heads) 175.9 ->
//     176.6.  The Step variant loses by it (786 -> 793 in a chain, 820 -> 839 behind a flush).
//   * Tensor cores do the dot products with the tokens on the M side so that G <= 8 query
//     heads fit the N=8 side without padding M: S^T[16 tok x 8 heads] = K[16 x D] Q^T[D x 8]
//     and O^T[D x 8] += V^T[D x 16] P^T[16 x 8] (mma.sync.m16n8k16, bf16 in / fp32 out).
//     The softmax statistics of a head are reduced over the 8 token lanes by warp shuffles.
//   * When a range leaves a sequence, the NW warps merge their (max, sum, O) through a
//     dedicated patch of shared memory.  A sequence that lies inside one range is normalised
//     and written as bf16 at once.  A sequence cut by a range boundary gives one fp32 partial
//     per range, written without waiting for anything; only its first and its last sequence can
//     be cut, so a block reports its (at most two) partials when its range is done.  The block
//     that reports the last partial (an arrival counter per (sequence, KV head) in the workspace,
//     no waiting) merges them in range order and writes the row, so there is no second launch.
//     The counters are returned to zero by that block.
//   * Step variant: the block that streams token ctx-1 of a sequence takes that row from the
//     new K/V activation instead of the cache (with the same asynchronous copies) and writes it to
//     its cache slot when the tile is used.  Layer variant: the same for any slot_mapping, a few rows.
//
// Small batches are bound by a chain of trips to memory: lengths, block table, K/V, then for cut
// sequences partials out, arrival, partials in.  Table lines are fetched under the lengths, the
// arrivals wait for nothing in the middle of a range, and a merge takes one trip for eight parts.
// Where parts are few they are written as marked cells (kMark), so that the report of a partial needs no fence and the
// merge's reads go out with it.
// One launch in a chain that stores the new rows too, from a graph (head_dim 128, 16 / 8 heads): one sequence of 300-600
// tokens 6.0 us, one of 4096 7.9, 8 of 100-1024 9.6, 16 of them 11.1, 64 of them 30.1; 256 sequences of 2048-8192
// tokens (32 / 8 heads) 745-755.
#include <cstdlib>
#include <type_traits>

#include "common.cuh"

// Pipeline shape of the head_dim-128 kernel: tokens per warp tile, ring stages per warp, warps per
// block (overridable at build time for sweeps; the defaults are the measured best).
#ifndef NVLLM_DEC_TT
#define NVLLM_DEC_TT 16
#endif
#ifndef NVLLM_DEC_NST
#define NVLLM_DEC_NST 3
#endif
#ifndef NVLLM_DEC_NW
#define NVLLM_DEC_NW 4
#endif

namespace nvllm {

// Workspace layout: [arrival counters: kCounterSlots u32][partials O][partials (max, sum)].
// The counter area has one fixed size so that calls of different geometries can share one
// workspace: whatever a call leaves in the partial area, the counters are all zero again.
constexpr int kCounterSlots = 16384;  // batch * Hkv must not exceed this
constexpr int64_t kCounterBytes = static_cast<int64_t>(kCounterSlots) * 4;
constexpr int kMaxDecodeCtas = 1024;  // the workspace is sized for at most this many thread blocks

struct DecodeParams {
  const __nv_bfloat16* q;
  int64_t q_stride;
  __nv_bfloat16* k_cache;  // written by the step and layer variants
  __nv_bfloat16* v_cache;
  const int32_t* ctx_lens;
  const int32_t* block_tables;
  int64_t bt_stride;
  int max_blocks;
  __nv_bfloat16* out;
  int64_t out_stride;
  int batch, hq, hkv, g;
  float scale_log2e;
  int64_t num_blocks;
  // step and layer variant: the new tokens' rows
  const __nv_bfloat16* k_new;
  int64_t k_new_stride;
  const __nv_bfloat16* v_new;
  int64_t v_new_stride;
  const int32_t* slot_mapping;
  int n_new;               // layer variant: new rows, one to a lane, stored to slot_mapping[row]
  int n_ranges;
  bool lengths_early;      // lengths and tables were complete before the previous kernel in the stream let this one start
  unsigned int* counters;  // [batch * hkv], zero between launches
  float* ws_o;             // [n_ranges + batch][hq][D]
  float* ws_ml;            // [n_ranges + batch][hq][2] = (running max in log2 units, sum)
  bool cells;              // partials as marked cells in ws_o: [n_ranges + batch][hq][D + 2] of 8 bytes, see kMark
  int* status;
};

template <int D_, int TT_, int NST_, int NW_>
struct DecodeCfg {
  static constexpr int D = D_, TT = TT_, NST = NST_, NW = NW_;
  static constexpr int UNIT = NW * TT;               // tokens per work unit
  static constexpr int CPR = D / 8;                  // 16-byte pieces per row
  static constexpr int ROW_BYTES = D * 2;
  static constexpr int TILE_BYTES = TT * ROW_BYTES;  // one tensor, one stage
  static constexpr int STAGE_BYTES = 2 * TILE_BYTES;
  static constexpr int WARP_BYTES = NST * STAGE_BYTES;
  static constexpr int RING_BYTES = NW * WARP_BYTES;
  static constexpr int MERGE_BYTES = NW * 8 * D * 4 + NW * 8 * 2 * 4;
  static constexpr int SMEM = RING_BYTES + MERGE_BYTES;
  static constexpr int MT = TT / 16;  // 16-token MMA row tiles per warp tile
  static constexpr int KS = D / 16;   // k-steps of the QK^T product
  static constexpr int DT = D / 16;   // 16-row tiles of O^T
  static_assert(TT % 16 == 0 && kBlockSize % TT == 0, "a warp tile must not straddle a cache block");
  static_assert((TT * CPR) % 32 == 0, "tile copy must divide evenly over a warp");
};

// Marked cells.  A word of a partial next to a mark, 8 bytes that are written and read as one: the block that merges
// sees for each of them whether it is there yet, so that a block that reports a partial needs no fence
// between the partial and its arrival, and one that may have been the last to arrive reads the others' while the
// answer is on its way.  What is read is marked only if it belongs to this launch: the block that merges takes the
// marks off again, and no other word in a workspace is ever this one: a workspace starts as zeros, and plain partials are
// results of single-precision arithmetic, whose only NaN is 0x7fffffff, whatever becomes of subnormal numbers.
constexpr uint32_t kMark = 0x7f99c3a7u;
static_assert((kMark & 0x7f800000u) == 0x7f800000u && (kMark & 0x007fffffu) != 0 && (kMark & 0x00400000u) == 0,
              "as a float a signalling NaN: no operation returns one");
constexpr int kMaxPolls = 1 << 20;  // the stores are on their way when a block polls for them: far more than it takes

__device__ __forceinline__ uint64_t cell(float x) { return static_cast<uint64_t>(kMark) << 32 | __float_as_uint(x); }
__device__ __forceinline__ bool marked(const ulonglong2& c) {
  return static_cast<uint32_t>(c.x >> 32) == kMark && static_cast<uint32_t>(c.y >> 32) == kMark;
}
__device__ __forceinline__ float value_of(uint64_t c) { return __uint_as_float(static_cast<uint32_t>(c)); }
__device__ __forceinline__ void store_cells(uint64_t* at, uint64_t a, uint64_t b) {
  asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(at), "l"(a), "l"(b) : "memory");
}
__device__ __forceinline__ ulonglong2 load_cells(const uint64_t* at) {
  ulonglong2 c;
  asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(c.x), "=l"(c.y) : "l"(at) : "memory");
  return c;
}

// The sequence a block is working in: index, global index of its first unit, units, length.
struct SeqCursor {
  int b, first, units, ctx;
  int slot;  // step variant: slot of the new token (-1: nothing is stored)
};

// A sequence whose units lie in several ranges: n of them, from r_first on.
struct Cut {
  int b, r_first, n;
};

// Cost of a streamed unit over the cost of a merged partial.  With merges of eight parts to a trip, us at 8 -> 16 -> 32: 36
// captured layers (32 / 8 heads) of two sequences of 500-4000 tokens 411 -> 358 -> 358, of one of 1050 281 -> 279 -> 289, of
// four of 100-1024 292.5 -> 294.5 -> 294.7; 28 (16 / 8 heads) of two of 500-4000 280 -> 264 -> 264; a layer of one of 4096 8.53 ->
// 8.12 -> 8.24.  At head_dim 64, where a merge has the statistics of 16 parts in a trip, 8 where 16 would cut a sequence into more
// than 32 parts (14 / 2 heads, layer of two of 20000-32000 tokens 57 parts 17.0, 41 parts 11.8; 7 / 1, six of 8000-16000 15.8, 12.3).
constexpr float kSplitBalance = 16.f, kSplitBalanceLong = 8.f;
constexpr int kSplitLong = 64;  // units of a sequence that make 32 parts at a balance of 16

// The kernels.  Step, StepGuess and Layer also store the new tokens' rows: the former two where the row's slot is that of its
// position, Layer to any slot.
// Guess, StepGuess and Layer make the first split of the batch, and the loads that follow from it, on lengths and table entries
// that the previous kernel may yet change (see where they branch).  In a chain of decode layers of 16 sequences, of
// which each streams 7 us, that takes the trips for lengths, sums, table and first rows off the path, and with
// nothing of Step in it the kernel starts its loads sooner: 17.4 -> 14.9 us a layer, 13.4 with the table and cells.
enum class Variant { Plain, Step, StepGuess, Guess, Layer };

template <class C, Variant V, bool CELLS>
__global__ void __launch_bounds__(C::NW * 32, 2) decode_paged_kernel(const DecodeParams p) {
  constexpr bool LAYER = V == Variant::Layer, STEP = V == Variant::Step || V == Variant::StepGuess;
  constexpr bool GUESS = V == Variant::Guess || V == Variant::StepGuess || LAYER;
  constexpr int D = C::D, TT = C::TT, NST = C::NST, NW = C::NW, UNIT = C::UNIT, NT = NW * 32;
  constexpr int QUADS = D / 4, GROUPS = NT / QUADS;  // lanes that hold a head four columns each; such groups in a block
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ int s_scan[NW];
  __shared__ int s_start[3];
  __shared__ int s_last_arrival[2];

  pdl_trigger();
  if (!GUESS && !p.lengths_early) pdl_wait();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int gid = lane >> 2, tig = lane & 3;
  const int kvh = blockIdx.x % p.hkv;
  const int range = blockIdx.x / p.hkv;
  const int ctx_cap = p.max_blocks * kBlockSize;
  auto capped = [&](int c) { return c < 0 ? 0 : (c > ctx_cap ? ctx_cap : c); };
  auto length_of = [&](int b) { return capped(p.ctx_lens[b]); };
  auto units_of = [](int ctx) { return (ctx + UNIT - 1) / UNIT; };
  auto write_zeros = [&](int b) {  // empty context: defined output, no cache access
    if (b % p.n_ranges != range) return;
    uint4* dst = reinterpret_cast<uint4*>(p.out + b * p.out_stride + static_cast<int64_t>(kvh * p.g) * D);
    for (int i = 0; i < p.g * D / 8; ++i) dst[i] = make_uint4(0u, 0u, 0u, 0u);
  };

  auto slot_of = [&](int b) { return STEP ? p.slot_mapping[b] : -1; };
  auto seek = [&](SeqCursor& c, int u) {  // u < total, so c.b stays inside the batch
    if (u < c.first + c.units) return;
    do {
      c.first += c.units;
      ++c.b;
      c.ctx = length_of(c.b);
      c.units = units_of(c.ctx);
    } while (u >= c.first + c.units && (!GUESS || c.b < p.batch - 1));  // a guess may count on more units than there are
    c.slot = slot_of(c.b);
  };

  // Q^T as the B operand: lane (gid, tig) holds q[head gid][16*ks + 2*tig .. +1] and [.. + 8].
  auto load_q = [&](uint32_t (&dst)[C::KS][2], int b) {
    const __nv_bfloat16* qrow = p.q + b * p.q_stride + static_cast<int64_t>(kvh * p.g + gid) * D;
#pragma unroll
    for (int ks = 0; ks < C::KS; ++ks) {
      if (gid < p.g) {
        dst[ks][0] = *reinterpret_cast<const uint32_t*>(qrow + ks * 16 + 2 * tig);
        dst[ks][1] = *reinterpret_cast<const uint32_t*>(qrow + ks * 16 + 8 + 2 * tig);
      } else {
        dst[ks][0] = 0u;
        dst[ks][1] = 0u;
      }
    }
  };

  const uint32_t warp_smem = smem_u32(smem) + warp * C::WARP_BYTES;
  const int64_t row_elems = static_cast<int64_t>(p.hkv) * D;

  int bad = 0;
  int new_slot = -1;   // layer variant, lane l: slot of the l-th new row
  unsigned fresh = 0;  // step variant: stages whose tile holds the new token's row
  auto load_rows = [&](int b, int t0, int ctx, int slot, int64_t blk, int stage) {
    const bool blk_ok = blk >= 0 && blk < p.num_blocks;
    if (!blk_ok) {
      bad |= NVLLM_STATUS_BAD_BLOCK;  // reported at the end: a guess may load for nothing
      blk = 0;
    }
    const int64_t slot0 = blk * kBlockSize + (t0 % kBlockSize);
    // Step variant: token ctx-1 is the one being decoded.  Its row comes from the activation,
    // provided slot_mapping agrees with the block table, and goes to the cache when the tile is used.
    const int last = ctx - 1;
    int new_row = -1;
    if (STEP && last < t0 + TT && slot >= 0) {  // last >= t0 holds because t0 < ctx
      if (blk_ok && slot == slot0 + (last - t0)) {
        new_row = last - t0;
        fresh |= 1u << stage;
      } else {
        bad |= NVLLM_STATUS_BAD_SLOT;
      }
    }
    // Layer variant: whatever row of whatever sequence lies in a slot that this launch stores to is the new
    // one, as it would be behind a launch that stores.
    unsigned stored = 0;
    if (LAYER && blk_ok) stored = __ballot_sync(0xffffffffu, new_slot >= slot0 && new_slot < slot0 + TT);
    const uint32_t kdst = warp_smem + stage * C::STAGE_BYTES;
    auto copy = [&](auto patch) {
#pragma unroll
      for (int it = 0; it < TT * C::CPR / 32; ++it) {
        const int idx = it * 32 + lane;
        const int r = idx / C::CPR, col = idx % C::CPR;
        const int bytes = (blk_ok && t0 + r < ctx) ? 16 : 0;
        const int64_t off = bytes ? (slot0 + r) * row_elems + kvh * D + col * 8 : 0;
        const __nv_bfloat16 *ksrc = p.k_cache + off, *vsrc = p.v_cache + off;
        if (STEP && r == new_row) {
          const int64_t in_row = static_cast<int64_t>(kvh) * D + col * 8;
          ksrc = p.k_new + b * p.k_new_stride + in_row;
          vsrc = p.v_new + b * p.v_new_stride + in_row;
        }
        if constexpr (decltype(patch)::value) {
          for (unsigned left = stored; left; left &= left - 1) {
            const int i = __ffs(left) - 1;
            if (__shfl_sync(0xffffffffu, new_slot, i) == slot0 + r) {
              ksrc = p.k_new + i * p.k_new_stride + kvh * D + col * 8;
              vsrc = p.v_new + i * p.v_new_stride + kvh * D + col * 8;
            }
          }
        }
        const uint32_t dst = kdst + r * C::ROW_BYTES + ((col ^ (r & 7)) << 4);
        cp_async16(dst, ksrc, bytes);
        cp_async16(dst + C::TILE_BYTES, vsrc, bytes);
      }
    };
    if (LAYER && stored) copy(std::true_type{});
    else copy(std::false_type{});
  };
  // ---- 1. units per sequence, block-wide scan, this block's range of the unit list ------
  const int per_thread = GUESS ? 1 : (p.batch + NT - 1) / NT;
  const int b_lo = min(tid * per_thread, p.batch), b_hi = min(b_lo + per_thread, p.batch);
  // The first table line of every sequence on its way to this SM while the lengths are summed: the
  // block does not know yet whose it needs (beyond this batch the stream hides the trip).
  auto prefetch_table = [&]() {
    if (p.batch <= NT && tid < p.batch)
      asm volatile("prefetch.global.L1 [%0];" ::"l"(p.block_tables + tid * p.bt_stride));
  };
  int total, n_ranges, per_range, longer, u0, u1, len_lo;
  int2* seqs = reinterpret_cast<int2*>(smem + C::RING_BYTES);  // a guess: first unit and length of every sequence
  static_assert(NT * 8 <= C::MERGE_BYTES, "room for them until the first merge");
  auto split = [&](bool ahead) {
    if (!GUESS) prefetch_table();
    int local = 0;
    len_lo = 0;
    for (int b = b_lo; b < b_hi; ++b) {
      const int c = ahead ? capped(__ldcg(p.ctx_lens + b)) : length_of(b);
      if (b == b_lo) len_lo = c;
      local += units_of(c);
      if (!GUESS && c == 0) write_zeros(b);
    }
    int incl = local;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += v;
    }
    if (lane == 31) s_scan[warp] = incl;
    __syncthreads();
    int before = 0;
    total = 0;
#pragma unroll
    for (int w = 0; w < NW; ++w) {
      if (w < warp) before += s_scan[w];
      total += s_scan[w];
    }
    const int excl = before + incl - local;
    if (GUESS && ahead) seqs[tid] = make_int2(excl, len_lo);
    // No more ranges than units, so that every range in use holds at least one unit and the ranges
    // that share a sequence are consecutive.  And where sequences are few, no more than balance the
    // two costs of a cut: a range streams total / n units and a sequence's merge reads n / batch
    // partials, so that the sum is least at n = sqrt(c total batch).
    const float balance = D == 64 && total > kSplitLong * p.batch ? kSplitBalanceLong : kSplitBalance;
    n_ranges = max(1, min(min(p.n_ranges, total), static_cast<int>(sqrtf(balance * total * p.batch))));
    if (range >= n_ranges || total == 0) return false;  // block-uniform (also when the whole batch is empty)
    // the first `longer` ranges hold one unit more than the others
    per_range = total / n_ranges, longer = total - per_range * n_ranges;
    u0 = range * per_range + min(range, longer);
    u1 = u0 + per_range + (range < longer ? 1 : 0);
    if (local > 0 && excl <= u0 && u0 < excl + local) {  // the one thread whose sequences hold unit u0
      int first = excl;
      for (int b = b_lo;; ++b) {
        const int len = b == b_lo ? len_lo : length_of(b), n = units_of(len);
        if (u0 < first + n) {
          s_start[0] = b;
          s_start[1] = first;
          s_start[2] = len;
          break;
        }
        first += n;
      }
    }
    __syncthreads();
    return true;
  };

  SeqCursor cc, pc;  // compute side; load side, NST-1 units ahead
  uint32_t qb[C::KS][2], qn[C::KS][2];  // this sequence's fragments; the next sequence's, fetched early
  int qn_b, n_units;
  // A guess: this warp's tiles of the range's first 32 units, one to a lane, -1 where it has no token in the unit.  Loaded
  // unrolled in a step only: its chain has no other kernel in it, and the code stays where it is (8 of 100-1024 11.4 rolled, 11.0).
  int n_listed = 0, listed_t0 = -1, listed_ctx = 0, listed_blk = 0, listed_b = 0, listed_slot = -1;
  auto load_unit = [&](int j) {  // the range's j-th unit, j < n_units, rising from call to call
    const int stage = j % NST;
    if (GUESS && j < n_listed) {
      const int t0 = __shfl_sync(0xffffffffu, listed_t0, j), ctx = __shfl_sync(0xffffffffu, listed_ctx, j);
      const int blk = __shfl_sync(0xffffffffu, listed_blk, j);
      const int b = STEP ? __shfl_sync(0xffffffffu, listed_b, j) : 0, slot = STEP ? __shfl_sync(0xffffffffu, listed_slot, j) : -1;
      if (STEP) fresh &= ~(1u << stage);
      if (t0 >= 0) load_rows(b, t0, ctx, slot, blk, stage);
      return;
    }
    seek(pc, u0 + j);
    fresh &= ~(1u << stage);
    const int t0 = (u0 + j - pc.first) * UNIT + warp * TT;
    if (t0 < pc.ctx) load_rows(pc.b, t0, pc.ctx, pc.slot, p.block_tables[pc.b * p.bt_stride + t0 / kBlockSize], stage);
  };
  auto start = [&]() {
    cc.b = s_start[0];
    cc.first = s_start[1];
    cc.ctx = s_start[2];
    cc.units = units_of(cc.ctx);
    cc.slot = slot_of(cc.b);
    pc = cc;
    if (!GUESS && p.lengths_early) pdl_wait();  // from here on the cache is read
    load_q(qb, cc.b);
    qn_b = min(cc.b + 1, p.batch - 1);
    load_q(qn, qn_b);
    n_units = u1 - u0;
#pragma unroll(GUESS && !STEP ? 1 : NST - 1)
    for (int j = 0; j < NST - 1; ++j) {
      if (j < n_units) load_unit(j);
      cp_async_commit();
    }
  };

  if constexpr (GUESS) {
    // The range is cut by what the lengths are now, its tiles are listed, one to a lane, with the table's entries as they
    // are now, and the first two units are brought to L2.  When the previous kernel is done those are loaded while
    // lengths and entries are read again, and if one has changed the range is cut anew.  What is read before the wait goes
    // round L1, is held to the bounds of the table and the cache, and serves the guess alone.  With the list no load of a
    // range waits for a length or a table entry (24 captured layers of 16 sequences, 14 / 2 heads of 64, 180 -> 166 us, a
    // layer of one of 317 tokens 6.25 -> 5.95).  Two units: with three or all of them the requests stand in the way of
    // the pre-attention step in front (28 layers of 16, 16 / 8 heads, 376 -> 393 and 415), with one the range starts
    // later (382).  The code itself is in the way of a launch that streams for 3 us: one copy of it for the guess and the
    // second attempt, rolled loops (36 layers of two sequences 509 -> 493).
    const int64_t n_slots = p.num_blocks * kBlockSize;
    auto in_cache = [&](int slot) { return slot >= 0 && slot < n_slots ? slot : -1; };
    if (LAYER && lane < p.n_new) new_slot = in_cache(__ldcg(p.slot_mapping + lane));
    int slot_now = -1;
    bool mine;
#pragma unroll 1
    for (bool ahead = true;; ahead = false) {
      mine = split(ahead);
      int now = 0, blk_now = 0, listed_slot_now = -1;
      if (ahead) {
        const int32_t* listed_at = p.block_tables;
        if (mine) {
          n_listed = min(u1 - u0, 32);
          if (lane < n_listed) {
            const int u = u0 + lane;
            int b = s_start[0];
            while (b + 1 < p.batch && u >= seqs[b].x + units_of(seqs[b].y)) ++b;
            const int t0 = (u - seqs[b].x) * UNIT + warp * TT;
            listed_ctx = seqs[b].y;
            if (t0 < listed_ctx) {
              listed_t0 = t0;
              listed_at += b * p.bt_stride + t0 / kBlockSize;
              listed_blk = __ldcg(listed_at);
              if (STEP) listed_b = b, listed_slot = __ldcg(p.slot_mapping + b);
            }
          }
#pragma unroll 1
          for (int j = 0; j < min(n_listed, NST - 1); ++j) {
            const int t0 = __shfl_sync(0xffffffffu, listed_t0, j), ctx = __shfl_sync(0xffffffffu, listed_ctx, j);
            const int64_t blk = __shfl_sync(0xffffffffu, listed_blk, j);
            if (t0 < 0 || blk < 0 || blk >= p.num_blocks) continue;
            constexpr int LINES = C::ROW_BYTES / 128;
#pragma unroll
            for (int it = 0; it < TT * LINES / 32; ++it) {
              const int r = (it * 32 + lane) / LINES, part = (it * 32 + lane) % LINES;
              const int64_t off = (blk * kBlockSize + t0 % kBlockSize + r) * row_elems + kvh * D + part * 64;
              if (t0 + r < ctx) {
                asm volatile("prefetch.global.L2 [%0];" ::"l"(p.k_cache + off));
                asm volatile("prefetch.global.L2 [%0];" ::"l"(p.v_cache + off));
              }
            }
          }
        }
        pdl_wait();
        if (tid < p.batch) now = length_of(tid);
        blk_now = listed_t0 >= 0 ? *listed_at : listed_blk;
        if (LAYER && lane < p.n_new) slot_now = p.slot_mapping[lane];
        if (STEP && listed_t0 >= 0) listed_slot_now = p.slot_mapping[listed_b];
      }
      if (mine) start();
      if (!ahead || !__syncthreads_or(now != len_lo || blk_now != listed_blk || (LAYER && in_cache(slot_now) != new_slot) || (STEP && listed_slot_now != listed_slot))) break;
      cp_async_wait<0>();
      __syncthreads();
      bad = 0;
      n_listed = 0;
      new_slot = in_cache(slot_now);
    }
    if (tid < p.batch && len_lo == 0) write_zeros(tid);
    if (LAYER && warp == NW - 1) {
      for (int i = range; i < p.n_new; i += p.n_ranges) {
        const int64_t slot = __shfl_sync(0xffffffffu, new_slot, i);
        if (slot < 0) continue;
        for (int k = lane; k < 2 * C::CPR; k += 32) {  // K pieces, then V pieces (for head_dim 128 one per lane)
          const bool is_k = k < C::CPR;
          const int64_t col = kvh * D + k % C::CPR * 8;
          *reinterpret_cast<uint4*>((is_k ? p.k_cache : p.v_cache) + slot * row_elems + col) =
              *reinterpret_cast<const uint4*>(is_k ? p.k_new + i * p.k_new_stride + col : p.v_new + i * p.v_new_stride + col);
        }
      }
      if (blockIdx.x == 0 && slot_now >= n_slots) atomicOr(p.status, NVLLM_STATUS_BAD_SLOT);
    }
    if (!mine) return;
  } else {
    if (!split(false)) {
      if (p.lengths_early) pdl_wait();  // every block waits: where all contexts are empty, none gets to start()
      return;
    }
    start();
  }
  // the range that holds global unit u
  auto range_of = [&](int u) {
    const int split = longer * (per_range + 1);
    return u < split ? u / (per_range + 1) : longer + (u - split) / per_range;
  };

  float o[C::DT][4];
  float m0, m1, l0, l1;  // heads 2*tig and 2*tig+1
  auto reset_state = [&]() {
#pragma unroll
    for (int dt = 0; dt < C::DT; ++dt) o[dt][0] = o[dt][1] = o[dt][2] = o[dt][3] = 0.f;
    m0 = m1 = -INFINITY;
    l0 = l1 = 0.f;
  };
  reset_state();

  float* sm_o = reinterpret_cast<float*>(smem + C::RING_BYTES);  // [NW][8][D]
  float* sm_ml = sm_o + NW * 8 * D;                              // [NW][8][2]

  auto add_scaled = [](float4& acc, const float4& v, float f) {
    acc.x += v.x * f;
    acc.y += v.y * f;
    acc.z += v.z * f;
    acc.w += v.w * f;
  };
  auto write_quad = [&](int b, int h, int d4, const float4& acc, float L) {
    const float inv = L > 0.f ? 1.f / L : 0.f;
    *reinterpret_cast<uint2*>(p.out + b * p.out_stride + static_cast<int64_t>(kvh * p.g + h) * D + d4 * 4) =
        make_uint2(pack_bf16x2(acc.x * inv, acc.y * inv), pack_bf16x2(acc.z * inv, acc.w * inv));
  };

  Cut cut0{}, cut1{};  // this range's sequences that other ranges share
  int n_cut = 0;
  // With cells every warp that writes some reports for itself.  Its first lane: how many had before it, at the last cut
  // and the one before that.  The former is not touched until it is needed, so that nothing waits for it.
  unsigned int arrived = 0, arrived0 = 0;
  const int writers = min(NW, (p.g * QUADS + 31) / 32);
  constexpr int HEAD_CELLS = D + 2;  // of a head's partial: D columns, maximum, sum
  auto cells_of = [&](int64_t slot, int h) {
    return reinterpret_cast<uint64_t*>(p.ws_o) + (slot * p.hq + kvh * p.g + h) * HEAD_CELLS;
  };

  // Leaves sequence cc.b: merges the NW warps' states and writes the output row or a partial.
  auto flush = [&]() {
#pragma unroll
    for (int sh = 4; sh <= 16; sh <<= 1) {
      l0 += __shfl_xor_sync(0xffffffffu, l0, sh);
      l1 += __shfl_xor_sync(0xffffffffu, l1, sh);
    }
    __syncthreads();  // the previous merge has been read by everyone
#pragma unroll
    for (int dt = 0; dt < C::DT; ++dt) {
      const int d = dt * 16 + gid;
      float* dst = sm_o + (warp * 8 + 2 * tig) * D + d;
      dst[0] = o[dt][0];
      dst[D] = o[dt][1];
      dst[8] = o[dt][2];
      dst[D + 8] = o[dt][3];
    }
    if (gid == 0) {
      sm_ml[(warp * 8 + 2 * tig) * 2 + 0] = m0;
      sm_ml[(warp * 8 + 2 * tig) * 2 + 1] = l0;
      sm_ml[(warp * 8 + 2 * tig + 1) * 2 + 0] = m1;
      sm_ml[(warp * 8 + 2 * tig + 1) * 2 + 1] = l1;
    }
    const int r_first = range_of(cc.first), r_last = range_of(cc.first + cc.units - 1);
    const int n_parts = r_last - r_first + 1;  // ranges that hold a piece of this sequence
    __syncthreads();
    for (int quad = tid; quad < p.g * QUADS; quad += NT) {  // four columns of a head per thread
      const int h = quad / QUADS, d4 = quad % QUADS;
      float m[NW], mm = -INFINITY, L = 0.f;
#pragma unroll
      for (int w = 0; w < NW; ++w) {
        m[w] = sm_ml[(w * 8 + h) * 2];
        mm = fmaxf(mm, m[w]);
      }
      float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int w = 0; w < NW; ++w) {
        const float f = m[w] == -INFINITY ? 0.f : fast_exp2(m[w] - mm);
        const float4 v = *reinterpret_cast<const float4*>(sm_o + (w * 8 + h) * D + d4 * 4);
        L += sm_ml[(w * 8 + h) * 2 + 1] * f;
        add_scaled(acc, v, f);
      }
      if (n_parts == 1) {
        write_quad(cc.b, h, d4, acc, L);
      } else {
        // partial slot range + b: strictly increasing along the (range, sequence) pieces of the list
        const int64_t row = static_cast<int64_t>(range + cc.b) * p.hq + kvh * p.g + h;
        if constexpr (CELLS) {
          uint64_t* to = cells_of(range + cc.b, h);
          store_cells(to + d4 * 4, cell(acc.x), cell(acc.y));
          store_cells(to + d4 * 4 + 2, cell(acc.z), cell(acc.w));
          if (d4 == 0) store_cells(to + D, cell(mm), cell(L));
        } else {
          *reinterpret_cast<float4*>(p.ws_o + row * D + d4 * 4) = acc;
          if (d4 == 0) *reinterpret_cast<float2*>(p.ws_ml + row * 2) = make_float2(mm, L);
        }
      }
    }
    if (n_parts > 1) {  // block-uniform
      if (n_cut == 0) cut0 = {cc.b, r_first, n_parts};
      else cut1 = {cc.b, r_first, n_parts};
      if (CELLS && warp < writers) {  // reported at once: the answer is looked at when the range is done
        __syncwarp();  // the warp's cells are on their way
        arrived0 = arrived;
        if (lane == 0)
          asm volatile("atom.relaxed.gpu.global.add.u32 %0, [%1], 1;" : "=r"(arrived) : "l"(p.counters + cc.b * p.hkv + kvh) : "memory");
      }
      ++n_cut;
    }
  };

  // Merges the partials of a cut sequence, all of which are in the workspace, and writes its rows.
  // QUADS lanes take a head (four columns each); lane l of them also holds the statistics of one
  // part of every chunk of QUADS parts, so that a chunk's statistics and its first rows are in
  // flight together and the weights go round by shuffle: a trip to L2 for every eight parts (when those past
  // the eighth were read one after the other, 17 parts of four heads took 7 us, and 36 captured layers of two sequences
  // of 500-4000 tokens 493 instead of 412; one layer of two of 32000, 14 / 2 heads of 64, 20.8 instead of 17.1).  Not through
  // shared memory by cp.async, all parts in one trip: 476 and 20.1, and one sequence of 350 tokens 193 -> 209.
  // Lane groups left over split the parts of a head between them.
  auto merge_cut = [&](const Cut& c) {
    constexpr int AHEAD = 8;
    const int group = tid / QUADS, gl = tid % QUADS;
    const int n_split = max(1, GROUPS / p.g);
    for (int h0 = 0; h0 < p.g; h0 += GROUPS) {
      const bool narrow = p.g < GROUPS;
      const int split = narrow ? group / p.g : 0, head = narrow ? group % p.g : min(h0 + group, p.g - 1);
      const bool active = narrow ? split < n_split : h0 + group < p.g;
      const int64_t row0 = static_cast<int64_t>(c.r_first + c.b) * p.hq + kvh * p.g + head;
      auto row_of = [&](int j) { return __ldcg(reinterpret_cast<const float4*>(p.ws_o + (row0 + static_cast<int64_t>(j) * p.hq) * D) + gl); };
      float mm = -INFINITY, L = 0.f;
      float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
      auto rebase = [&](float m_new) {
        const float keep = mm == -INFINITY ? 0.f : fast_exp2(mm - m_new);
        L *= keep;
        acc.x *= keep;
        acc.y *= keep;
        acc.z *= keep;
        acc.w *= keep;
        mm = m_new;
      };
      for (int j0 = 0; j0 < c.n; j0 += QUADS * n_split) {  // block-uniform; a group's parts are split + n_split * k
        float4 rows[AHEAD];
#pragma unroll
        for (int k = 0; k < AHEAD; ++k) {
          const int j = j0 + k * n_split + split;
          if (active && j < c.n) rows[k] = row_of(j);
        }
        const int mine = j0 + gl * n_split + split;
        float2 ml = make_float2(-INFINITY, 0.f);
        if (active && mine < c.n)
          ml = __ldcg(reinterpret_cast<const float2*>(p.ws_ml + (row0 + static_cast<int64_t>(mine) * p.hq) * 2));
        float m_new = fmaxf(mm, ml.x);
#pragma unroll
        for (int sh = QUADS / 2; sh > 0; sh >>= 1) m_new = fmaxf(m_new, __shfl_xor_sync(0xffffffffu, m_new, sh));
        rebase(m_new);
        const float f = ml.x == -INFINITY ? 0.f : fast_exp2(ml.x - m_new);
        float sum = ml.y * f;
#pragma unroll
        for (int sh = QUADS / 2; sh > 0; sh >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, sh);
        L += sum;
#pragma unroll
        for (int k = 0; k < AHEAD; ++k) {
          const float fk = __shfl_sync(0xffffffffu, f, k, QUADS);
          if (active && j0 + k * n_split + split < c.n) add_scaled(acc, rows[k], fk);
        }
        const int n_here = min(QUADS, (c.n - j0 + n_split - 1) / n_split);
#pragma unroll 1
        for (int k0 = AHEAD; k0 < n_here; k0 += AHEAD) {
#pragma unroll
          for (int k = 0; k < AHEAD; ++k) {
            const int j = j0 + (k0 + k) * n_split + split;
            if (active && j < c.n) rows[k] = row_of(j);
          }
#pragma unroll
          for (int k = 0; k < AHEAD; ++k) {
            const float fk = __shfl_sync(0xffffffffu, f, k0 + k, QUADS);
            if (active && j0 + (k0 + k) * n_split + split < c.n) add_scaled(acc, rows[k], fk);
          }
        }
      }
      if (n_split > 1) {  // block-uniform
        float* patch = sm_o + group * (D + 4);
        if (active && split > 0) {
          *reinterpret_cast<float4*>(patch + gl * 4) = acc;
          if (gl == 0) *reinterpret_cast<float2*>(patch + D) = make_float2(mm, L);
        }
        __syncthreads();
        if (active && split == 0)
          for (int k = 1; k < n_split; ++k) {
            const float* other = sm_o + (group + k * p.g) * (D + 4);
            const float2 ml = *reinterpret_cast<const float2*>(other + D);
            rebase(fmaxf(mm, ml.x));
            const float f = ml.x == -INFINITY ? 0.f : fast_exp2(ml.x - mm);
            L += ml.y * f;
            add_scaled(acc, *reinterpret_cast<const float4*>(other + gl * 4), f);
          }
        __syncthreads();
      }
      if (active && split == 0) write_quad(c.b, head, gl, acc, L);
    }
    if (tid == 0) p.counters[c.b * p.hkv + kvh] = 0u;  // ready for the next launch
  };

  // The same from cells, of both cuts, the one reported last first: its first reads are issued before it is known whether
  // this block was the last to arrive.  Rolled up: this is run once, and its instructions are on the way to the end.
  auto merge_cells = [&]() {
    constexpr int AHEAD = 8;
    const int group = tid / QUADS, gl = tid % QUADS;
    const int n_split = max(1, GROUPS / p.g);
    const bool narrow = p.g < GROUPS;
    const int split = narrow ? group / p.g : 0;
    const int64_t next = static_cast<int64_t>(p.hq) * HEAD_CELLS * n_split;  // from a part to the next one of this group's
    int polls = 0;
    auto was_last = [&](unsigned int before, const Cut& c) { return lane == 0 && warp < writers && before == static_cast<unsigned int>(c.n * writers - 1); };
    const bool first_to_merge = n_cut > 1 && __syncthreads_or(was_last(arrived0, cut0));
#pragma unroll 1
    for (int which = n_cut - 1; which >= 0; --which) {
      const Cut c = which ? cut1 : cut0;
      bool ask = which == n_cut - 1;
      if (!ask && !first_to_merge) break;
#pragma unroll 1
      for (int h0 = 0; h0 < p.g; h0 += GROUPS) {
        const int head = narrow ? group % p.g : min(h0 + group, p.g - 1);
        const bool active = narrow ? split < n_split : h0 + group < p.g;
        // the parts of a group: split, split + n_split and so on
        const int parts = active && c.n > split ? (c.n - split + n_split - 1) / n_split : 0;
        uint64_t* const from = cells_of(c.r_first + c.b, head) + split * static_cast<int64_t>(p.hq) * HEAD_CELLS;
        float mm = -INFINITY, L = 0.f, f = 0.f;
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        auto rebase = [&](float m_new) {
          const float keep = mm == -INFINITY ? 0.f : fast_exp2(mm - m_new);
          L *= keep;
          acc.x *= keep;
          acc.y *= keep;
          acc.z *= keep;
          acc.w *= keep;
          mm = m_new;
        };
        const int rounds = (c.n + n_split - 1) / n_split;  // of the group with most parts
#pragma unroll 1
        for (int k0 = 0; k0 < rounds; k0 += AHEAD) {
          // a lane holds the statistics of one of QUADS parts, and four columns of AHEAD of them
          const bool fresh_ml = k0 % QUADS == 0, have = fresh_ml && k0 + gl < parts;
          ulonglong2 ml = make_ulonglong2(0, 0), lo[AHEAD], hi[AHEAD];
          uint64_t* const ml_at = from + (k0 + gl) * next + D;
          uint64_t* const row_at = from + k0 * next + gl * 4;
          bool there;
          do {
            there = true;
            if (have) ml = load_cells(ml_at);
#pragma unroll
            for (int k = 0; k < AHEAD; ++k)
              if (k0 + k < parts) {
                lo[k] = load_cells(row_at + k * next);
                hi[k] = load_cells(row_at + k * next + 2);
              }
            if (ask) {  // block-uniform
              ask = false;
              if (!__syncthreads_or(was_last(arrived, c))) goto next_cut;
            }
            if (have) there = marked(ml);
#pragma unroll
            for (int k = 0; k < AHEAD; ++k)
              if (k0 + k < parts) there = there && marked(lo[k]) && marked(hi[k]);
          } while (!there && ++polls < kMaxPolls);
          if (fresh_ml) {
            const float m_mine = have ? value_of(ml.x) : -INFINITY;
            float m_new = fmaxf(mm, m_mine);
#pragma unroll
            for (int sh = QUADS / 2; sh > 0; sh >>= 1) m_new = fmaxf(m_new, __shfl_xor_sync(0xffffffffu, m_new, sh));
            rebase(m_new);
            f = m_mine == -INFINITY ? 0.f : fast_exp2(m_mine - m_new);
            float sum = have ? value_of(ml.y) * f : 0.f;
#pragma unroll
            for (int sh = QUADS / 2; sh > 0; sh >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, sh);
            L += sum;
            if (have) store_cells(ml_at, 0, 0);
          }
#pragma unroll
          for (int k = 0; k < AHEAD; ++k) {
            const float fk = __shfl_sync(0xffffffffu, f, (k0 + k) % QUADS, QUADS);
            if (k0 + k >= parts) continue;
            add_scaled(acc, make_float4(value_of(lo[k].x), value_of(lo[k].y), value_of(hi[k].x), value_of(hi[k].y)), fk);
            store_cells(row_at + k * next, 0, 0);
            store_cells(row_at + k * next + 2, 0, 0);
          }
        }
        if (n_split > 1) {  // block-uniform
          float* patch = sm_o + group * (D + 4);
          if (active && split > 0) {
            *reinterpret_cast<float4*>(patch + gl * 4) = acc;
            if (gl == 0) *reinterpret_cast<float2*>(patch + D) = make_float2(mm, L);
          }
          __syncthreads();
          if (active && split == 0)
            for (int k = 1; k < n_split; ++k) {
              const float* other = sm_o + (group + k * p.g) * (D + 4);
              const float2 ml = *reinterpret_cast<const float2*>(other + D);
              rebase(fmaxf(mm, ml.x));
              const float fo = ml.x == -INFINITY ? 0.f : fast_exp2(ml.x - mm);
              L += ml.y * fo;
              add_scaled(acc, *reinterpret_cast<const float4*>(other + gl * 4), fo);
            }
        }
        if (active && split == 0) write_quad(c.b, head, gl, acc, L);
      }
      if (tid == 0) p.counters[c.b * p.hkv + kvh] = 0u;  // ready for the next launch
    next_cut:
      __syncthreads();  // the patch and the answer have been read
    }
    if (polls >= kMaxPolls) atomicOr(p.status, NVLLM_STATUS_TIMEOUT);
  };

  // ---- 2. stream the range ------------------------------------------------------------------
  for (int i = 0;; ++i) {
    const int u = u0 + i;
    if (i == n_units || u >= cc.first + cc.units) {  // block-uniform: the range leaves sequence cc.b
      flush();
      if (i == n_units) break;
      seek(cc, u);
      reset_state();
      if (qn_b == cc.b) {
#pragma unroll
        for (int ks = 0; ks < C::KS; ++ks) {
          qb[ks][0] = qn[ks][0];
          qb[ks][1] = qn[ks][1];
        }
      } else {  // empty sequences in between
        load_q(qb, cc.b);
      }
      qn_b = min(cc.b + 1, p.batch - 1);
      load_q(qn, qn_b);
    }
    cp_async_wait<NST - 2>();
    if (V == Variant::Plain) __syncthreads();  // the warps' tiles of a unit are fetched together
    else __syncwarp();
    if (i + NST - 1 < n_units) load_unit(i + NST - 1);
    cp_async_commit();

    const int t0 = (u - cc.first) * UNIT + warp * TT;
    if (t0 >= cc.ctx) continue;
    const int t_end = cc.ctx;
    const uint32_t kbase = warp_smem + (i % NST) * C::STAGE_BYTES;
    const uint32_t vbase = kbase + C::TILE_BYTES;
    if (fresh >> (i % NST) & 1u) {  // step variant: the new token's row, on its way to the cache
      const int r = cc.ctx - 1 - t0;
      if (lane < 2 * C::CPR) {  // K pieces, then V pieces (for head_dim 128 one per lane)
        const int col = lane % C::CPR;
        const uint4 v = ld_shared16((lane < C::CPR ? kbase : vbase) + r * C::ROW_BYTES + ((col ^ (r & 7)) << 4));
        *reinterpret_cast<uint4*>((lane < C::CPR ? p.k_cache : p.v_cache) + static_cast<int64_t>(cc.slot) * row_elems + kvh * D +
                                  col * 8) = v;
      }
    }

    // S^T = K Q^T
    float s[C::MT][4];
#pragma unroll
    for (int mt = 0; mt < C::MT; ++mt) {
      s[mt][0] = s[mt][1] = s[mt][2] = s[mt][3] = 0.f;
      const int r = mt * 16 + (lane & 7) + ((lane >> 3) & 1) * 8;
#pragma unroll
      for (int ks = 0; ks < C::KS; ++ks) {
        const int c = ks * 2 + (lane >> 4);
        uint32_t a0, a1, a2, a3;
        ldmatrix_x4(a0, a1, a2, a3, kbase + r * C::ROW_BYTES + ((c ^ (r & 7)) << 4));
        mma_bf16_16816(s[mt], a0, a1, a2, a3, qb[ks][0], qb[ks][1]);
      }
    }

    // scale into log2 units, mask the tail, running max / sum per head
    const bool tail = t0 + TT > t_end;
    float mx0 = -INFINITY, mx1 = -INFINITY;
#pragma unroll
    for (int mt = 0; mt < C::MT; ++mt) {
#pragma unroll
      for (int e = 0; e < 4; ++e) s[mt][e] *= p.scale_log2e;
      if (tail) {
        const int tr = t0 + mt * 16 + gid;
        if (tr >= t_end) s[mt][0] = s[mt][1] = -INFINITY;
        if (tr + 8 >= t_end) s[mt][2] = s[mt][3] = -INFINITY;
      }
      mx0 = fmaxf(mx0, fmaxf(s[mt][0], s[mt][2]));
      mx1 = fmaxf(mx1, fmaxf(s[mt][1], s[mt][3]));
    }
#pragma unroll
    for (int sh = 4; sh <= 16; sh <<= 1) {
      mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, sh));
      mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, sh));
    }
    const float mn0 = fmaxf(m0, mx0), mn1 = fmaxf(m1, mx1);  // finite: the tile has >= 1 live token
    const float alpha0 = fast_exp2(m0 - mn0), alpha1 = fast_exp2(m1 - mn1);
    m0 = mn0;
    m1 = mn1;
    float ps0 = 0.f, ps1 = 0.f;
#pragma unroll
    for (int mt = 0; mt < C::MT; ++mt) {
      s[mt][0] = fast_exp2(s[mt][0] - mn0);
      s[mt][1] = fast_exp2(s[mt][1] - mn1);
      s[mt][2] = fast_exp2(s[mt][2] - mn0);
      s[mt][3] = fast_exp2(s[mt][3] - mn1);
      ps0 += s[mt][0] + s[mt][2];
      ps1 += s[mt][1] + s[mt][3];
    }
    l0 = l0 * alpha0 + ps0;  // per-lane partial sums; reduced over the token lanes at the flush
    l1 = l1 * alpha1 + ps1;
#pragma unroll
    for (int dt = 0; dt < C::DT; ++dt) {
      o[dt][0] *= alpha0;
      o[dt][1] *= alpha1;
      o[dt][2] *= alpha0;
      o[dt][3] *= alpha1;
    }

    // O^T += V^T P^T
#pragma unroll
    for (int mt = 0; mt < C::MT; ++mt) {
      const uint32_t pb0 = movmatrix_trans(pack_bf16x2(s[mt][0], s[mt][1]));
      const uint32_t pb1 = movmatrix_trans(pack_bf16x2(s[mt][2], s[mt][3]));
      const int r = mt * 16 + (lane & 7) + (lane >> 4) * 8;
#pragma unroll
      for (int dt = 0; dt < C::DT; ++dt) {
        const int c = dt * 2 + ((lane >> 3) & 1);
        uint32_t a0, a1, a2, a3;
        ldmatrix_x4_trans(a0, a1, a2, a3, vbase + r * C::ROW_BYTES + ((c ^ (r & 7)) << 4));
        mma_bf16_16816(o[dt], a0, a1, a2, a3, pb0, pb1);
      }
    }
  }
  cp_async_wait<0>();
  if (bad && lane == 0) atomicOr(p.status, bad);
  if (n_cut == 0) return;  // block-uniform
  if constexpr (CELLS) {
    merge_cells();
    return;
  }
  __syncthreads();         // every thread's partials are written
  if (tid < n_cut) {
    const Cut& c = tid == 0 ? cut0 : cut1;
    unsigned int before;  // releases the block's partials (the barrier ordered them before), acquires the others'
    asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;"
                 : "=r"(before) : "l"(p.counters + c.b * p.hkv + kvh) : "memory");
    s_last_arrival[tid] = before == static_cast<unsigned int>(c.n - 1);
  }
  __syncthreads();
  if (s_last_arrival[0]) merge_cut(cut0);
  if (n_cut > 1 && s_last_arrival[1]) merge_cut(cut1);
}

// ---- host side -------------------------------------------------------------------------

static int env_int(const char* name, int dflt) {
  const char* s = std::getenv(name);
  if (!s || !*s) return dflt;
  return std::atoi(s);
}

// Thread blocks of a launch: two per SM of the current device (NVLLM_DECODE_CTAS, read once per
// process, overrides the total for measurements), at most kMaxDecodeCtas; with no usable device
// the cap itself, so that the sizing functions work on any host.
static int decode_ctas() {
  static const int forced = env_int("NVLLM_DECODE_CTAS", 0);
  int n = forced > 0 ? forced : 2 * num_sms();
  if (n <= 0 || n > kMaxDecodeCtas) n = kMaxDecodeCtas;
  return n;
}
static int ranges_for(int ctas, int hkv) {
  const int n = ctas / hkv;
  return n < 1 ? 1 : n;
}
static int unit_tokens(int d) { return d == 128 ? NVLLM_DEC_NW * NVLLM_DEC_TT : 4 * 32; }

static int check_decode_geometry(const char* who, int batch, int max_blocks, int hq, int hkv, int d) {
  if (d != 64 && d != 128) return fail(NVLLM_E_GEOMETRY, "%s: head_dim=%d unsupported (64 or 128)", who, d);
  if (hq <= 0 || hkv <= 0 || hq % hkv) return fail(NVLLM_E_GEOMETRY, "%s: Hq=%d must be a positive multiple of Hkv=%d", who, hq, hkv);
  if (hq / hkv > 8) return fail(NVLLM_E_GEOMETRY, "%s: group size Hq/Hkv=%d > 8 unsupported", who, hq / hkv);
  if (batch < 0 || max_blocks <= 0) return fail(NVLLM_E_GEOMETRY, "%s: batch=%d max_blocks=%d invalid", who, batch, max_blocks);
  if (static_cast<int64_t>(batch) * hkv > kCounterSlots)
    return fail(NVLLM_E_GEOMETRY, "%s: batch*Hkv=%lld exceeds the %d (sequence, KV head) pairs of one launch", who,
                (long long)batch * hkv, kCounterSlots);
  // the unit list of a launch is indexed with 32-bit integers
  const int64_t max_units = (static_cast<int64_t>(max_blocks) * kBlockSize + unit_tokens(d) - 1) / unit_tokens(d);
  if (static_cast<int64_t>(max_blocks) * kBlockSize > 0x7fffffffLL || max_units * (batch > 0 ? batch : 1) > 0x3fffffffLL)
    return fail(NVLLM_E_GEOMETRY, "%s: batch=%d x max_blocks=%d too large", who, batch, max_blocks);
  return NVLLM_OK;
}

// Counter area plus one partial per (range, sequence) piece of the unit list; there are fewer
// than ranges + batch pieces.  Sized for the cap on thread blocks, not for the device at hand.
static int64_t workspace_bytes_for(int batch, int hq, int hkv, int d) {
  if (batch == 0) return 0;
  const int64_t rows = (static_cast<int64_t>(ranges_for(kMaxDecodeCtas, hkv)) + batch) * hq;
  return kCounterBytes + rows * d * 4 + rows * 2 * 4;
}

template <class C>
static int launch_decode(const DecodeParams& p, cudaStream_t stream) {
  constexpr bool HAS_CELLS = C::D == 128;
  // All variants at once; those with cells when the first of them is launched (loading a kernel costs the process about a
  // millisecond).  That may be inside a capture.
  static bool attr_set[2][64] = {{false}};
  int dev = 0;
  cudaGetDevice(&dev);
  auto reserve = [](auto cells) {
    constexpr bool K = decltype(cells)::value;
    for (auto kernel : {decode_paged_kernel<C, Variant::Plain, K>, decode_paged_kernel<C, Variant::Step, K>, decode_paged_kernel<C, Variant::StepGuess, K>,
                        decode_paged_kernel<C, Variant::Guess, K>, decode_paged_kernel<C, Variant::Layer, K>}) {
      const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM);
      if (e != cudaSuccess) return fail(NVLLM_E_CUDA, "decode_paged: cannot reserve %d bytes of shared memory: %s", C::SMEM, cudaGetErrorString(e));
    }
    return NVLLM_OK;
  };
  if (dev >= 0 && dev < 64 && !attr_set[p.cells][dev]) {
    const int rc = p.cells ? reserve(std::bool_constant<HAS_CELLS>{}) : reserve(std::false_type{});
    if (rc) return rc;
    attr_set[p.cells][dev] = true;
  }
  // A guess for launches with a sequence per thread at most.  Larger batches stream long enough for the trips
  // at the start not to matter.  Steps without and with it, us: 16 / 8 heads, one sequence of 317 tokens 6.6 -> 6.2, 8 of 100-1024
  // 11.2 -> 11.0, 32 19.9 -> 18.4, 100 43.4 -> 41.6, 128 53.1 -> 50.8; 32 / 8 heads, 6 of 205-405 7.15 -> 6.55, 54 of 587-1349 40.1 ->
  // 38.9; 14 / 2 heads of 64, 16 of 100-1024 7.0 -> 6.3, 8 of 8000-32000 26.1 -> 22.6.
  const Variant v = p.n_new > 0                                 ? Variant::Layer
                    : p.k_new && p.batch <= C::NW * 32            ? Variant::StepGuess
                    : p.k_new                                   ? Variant::Step
                    : !p.lengths_early && p.batch <= C::NW * 32 ? Variant::Guess
                                                                : Variant::Plain;
  auto pick = [v](auto cells) {
    constexpr bool K = decltype(cells)::value;
    return v == Variant::Layer   ? decode_paged_kernel<C, Variant::Layer, K>
           : v == Variant::Step  ? decode_paged_kernel<C, Variant::Step, K>
           : v == Variant::StepGuess ? decode_paged_kernel<C, Variant::StepGuess, K>
           : v == Variant::Guess ? decode_paged_kernel<C, Variant::Guess, K>
                                 : decode_paged_kernel<C, Variant::Plain, K>;
  };
  auto kernel = p.cells ? pick(std::bool_constant<HAS_CELLS>{}) : pick(std::false_type{});
  const int grid = p.n_ranges * p.hkv;
  return launch_kernel("decode_paged", kernel,
                       dim3(static_cast<unsigned>(grid)), dim3(C::NW * 32), C::SMEM, stream, p);
}

// Shared body of nvllm_decode_paged and nvllm_decode_step.
static int decode_common(const char* who, const void* q, int64_t q_row_stride, const void* k_new, int64_t k_new_row_stride,
                         const void* v_new, int64_t v_new_row_stride, const int32_t* slot_mapping, void* k_cache,
                         void* v_cache, const int32_t* context_lens, const int32_t* block_tables, int64_t bt_row_stride,
                         int32_t max_blocks, void* out, int64_t out_row_stride, int32_t batch, int32_t num_q_heads,
                         int32_t num_kv_heads, int32_t head_dim, float scale, int64_t num_blocks, void* workspace,
                         int64_t workspace_bytes, void* stream, bool with_store, bool lengths_early, int n_new = 0) {
  int rc = check_decode_geometry(who, batch, max_blocks, num_q_heads, num_kv_heads, head_dim);
  if (rc) return rc;
  if (batch == 0) return NVLLM_OK;
  if (!q || !k_cache || !v_cache || !context_lens || !block_tables || !out)
    return fail(NVLLM_E_NULL, "%s: NULL pointer argument", who);
  if (num_blocks <= 0) return fail(NVLLM_E_GEOMETRY, "%s: num_blocks=%lld must be positive", who, (long long)num_blocks);
  const int64_t qrow = static_cast<int64_t>(num_q_heads) * head_dim;
  const int64_t kvrow = static_cast<int64_t>(num_kv_heads) * head_dim;
  if (q_row_stride < qrow || out_row_stride < qrow || bt_row_stride < max_blocks)
    return fail(NVLLM_E_GEOMETRY, "%s: a row stride is smaller than its row", who);
  if (q_row_stride % 8 || out_row_stride % 8 || !aligned16(q) || !aligned16(out) || !aligned16(k_cache) || !aligned16(v_cache))
    return fail(NVLLM_E_ALIGN, "%s: q/out/cache pointers and row strides must be 16-byte aligned", who);
  if (with_store) {
    if (!k_new || !v_new || !slot_mapping) return fail(NVLLM_E_NULL, "%s: NULL pointer argument", who);
    if (k_new_row_stride < kvrow || v_new_row_stride < kvrow)
      return fail(NVLLM_E_GEOMETRY, "%s: key/value row stride smaller than Hkv*D", who);
    if (k_new_row_stride % 8 || v_new_row_stride % 8 || !aligned16(k_new) || !aligned16(v_new))
      return fail(NVLLM_E_ALIGN, "%s: key/value pointers and row strides must be 16-byte aligned", who);
  }
  const int64_t need = workspace_bytes_for(batch, num_q_heads, num_kv_heads, head_dim);
  if (!workspace || workspace_bytes < need)
    return fail(NVLLM_E_WORKSPACE, "%s: workspace of %lld bytes needed, %lld given", who, (long long)need,
                (long long)(workspace ? workspace_bytes : 0));
  if (!aligned16(workspace)) return fail(NVLLM_E_ALIGN, "%s: workspace must be 16-byte aligned", who);

  DecodeParams p;
  p.status = status_word();
  if (!p.status) return fail(NVLLM_E_NO_DEVICE, "%s: no CUDA device is usable", who);
  p.q = static_cast<const __nv_bfloat16*>(q);
  p.q_stride = q_row_stride;
  p.k_cache = static_cast<__nv_bfloat16*>(k_cache);
  p.v_cache = static_cast<__nv_bfloat16*>(v_cache);
  p.ctx_lens = context_lens;
  p.block_tables = block_tables;
  p.bt_stride = bt_row_stride;
  p.max_blocks = max_blocks;
  p.out = static_cast<__nv_bfloat16*>(out);
  p.out_stride = out_row_stride;
  p.batch = batch;
  p.hq = num_q_heads;
  p.hkv = num_kv_heads;
  p.g = num_q_heads / num_kv_heads;
  p.scale_log2e = scale * 1.4426950408889634f;
  p.num_blocks = num_blocks;
  p.k_new = with_store ? static_cast<const __nv_bfloat16*>(k_new) : nullptr;
  p.k_new_stride = k_new_row_stride;
  p.v_new = with_store ? static_cast<const __nv_bfloat16*>(v_new) : nullptr;
  p.v_new_stride = v_new_row_stride;
  p.slot_mapping = slot_mapping;
  p.n_new = n_new;
  p.lengths_early = lengths_early;
  p.n_ranges = ranges_for(decode_ctas(), num_kv_heads);
  const int64_t rows = (static_cast<int64_t>(ranges_for(kMaxDecodeCtas, num_kv_heads)) + batch) * num_q_heads;
  p.counters = static_cast<unsigned int*>(workspace);
  p.ws_o = reinterpret_cast<float*>(static_cast<unsigned char*>(workspace) + kCounterBytes);
  p.ws_ml = p.ws_o + rows * head_dim;
  // Marked cells, where a sequence is cut into few parts of few bytes: else the doubled bytes and the reads for nothing
  // cost more than the fence.  How many parts there are depends on lengths that only the device has; where a range has two
  // or three units of a chain of layers, cells lose 1-2 %, so that the line is one of averages.  us for 28 captured
  // layers of 2 query heads to a KV head, without -> with, by KV heads (ranges), batch and tokens:
  //   8 (37)    13 of 12-100 214 -> 205, of 64-512 315 -> 290, of 100-1024 382 -> 368, of 375-3000 566 -> 551; 16 214 -> 208, 348 ->
  //             356, 416 -> 391, 667 -> 647; 24 221 -> 214, 372 -> 380, 488 -> 473; 54 311 -> 281, 517 -> 492
  //   4 (74)    25 205 -> 199, 310 -> 301, 372 -> 370, 560 -> 549; 32 of 64-512 335 -> 341; 48 218 -> 210, 364 -> 366, 457 -> 445;
  //             108 307 -> 285, 524 -> 497
  //   2 (148)   50 208 -> 201, 307 -> 303, 361 -> 366, 543 -> 527; 96 215 -> 208, 360 -> 364, 465 -> 440; 216 344 -> 322, 566 -> 537
  //   1 (296)   99 211 -> 203, 312 -> 303, 359 -> 367, 563 -> 543; 256 317 -> 297, 471 -> 453, 604 -> 581; 400 351 -> 328, 828 -> 793
  // The step variant gains everywhere (1-10 %; 16 of 64-512, 8 KV heads, 11.1 -> 10.3 us, 50 of them, 2 KV heads, 10.1 -> 9.2).  A
  // layer with its store: 8 sequences of 100-1024 10.25 -> 11.4, 24 of 66-200 10.95 -> 11.5; 30-32 of 12-100 7.4 -> 7.4, of
  // 64-512 14.2 -> 13.5, of 100-1024 19.2 -> 18.3.  4 query heads to a KV head: 36 captured layers of 16 541 -> 547.  Cells take
  // twice the room; the workspace is sized for more thread blocks than this device takes, so that those of up to
  // 400 / Hkv sequences fit all the same.
  p.cells = (n_new > 0 ? 4 * p.n_ranges <= 5 * batch : p.n_ranges <= 3 * batch) && p.g <= 2 && head_dim == 128 &&
            (p.n_ranges + static_cast<int64_t>(batch)) * num_q_heads * 2 <= rows;

  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (head_dim == 128) return launch_decode<DecodeCfg<128, NVLLM_DEC_TT, NVLLM_DEC_NST, NVLLM_DEC_NW>>(p, st);
  return launch_decode<DecodeCfg<64, 32, 3, 4>>(p, st);
}

}  // namespace nvllm

extern "C" int64_t nvllm_decode_workspace_bytes(int32_t batch, int32_t max_blocks, int32_t num_q_heads,
                                                int32_t num_kv_heads, int32_t head_dim) {
  using namespace nvllm;
  int rc = check_decode_geometry("decode_workspace_bytes", batch, max_blocks, num_q_heads, num_kv_heads, head_dim);
  if (rc) return rc;
  return workspace_bytes_for(batch, num_q_heads, num_kv_heads, head_dim);
}

extern "C" int nvllm_decode_plan(int32_t batch, int32_t max_blocks, int32_t num_q_heads, int32_t num_kv_heads,
                                 int32_t head_dim, int32_t* unit_tokens_out, int32_t* thread_blocks_out) {
  using namespace nvllm;
  int rc = check_decode_geometry("decode_plan", batch, max_blocks, num_q_heads, num_kv_heads, head_dim);
  if (rc) return rc;
  if (unit_tokens_out) *unit_tokens_out = unit_tokens(head_dim);
  if (thread_blocks_out) *thread_blocks_out = ranges_for(decode_ctas(), num_kv_heads) * num_kv_heads;
  return NVLLM_OK;
}

extern "C" int nvllm_decode_paged(const void* q, int64_t q_row_stride, const void* k_cache, const void* v_cache,
                                  const int32_t* context_lens, const int32_t* block_tables, int64_t bt_row_stride,
                                  int32_t max_blocks, void* out, int64_t out_row_stride, int32_t batch,
                                  int32_t num_q_heads, int32_t num_kv_heads, int32_t head_dim, float scale,
                                  int64_t num_blocks, void* workspace, int64_t workspace_bytes, void* stream) {
  return nvllm::decode_common("decode_paged", q, q_row_stride, nullptr, 0, nullptr, 0, nullptr, const_cast<void*>(k_cache),
                              const_cast<void*>(v_cache), context_lens, block_tables, bt_row_stride, max_blocks, out,
                              out_row_stride, batch, num_q_heads, num_kv_heads, head_dim, scale, num_blocks, workspace,
                              workspace_bytes, stream, false, false);
}

extern "C" int nvllm_decode_step(const void* q, int64_t q_row_stride, const void* key, int64_t key_row_stride,
                                 const void* value, int64_t value_row_stride, const int32_t* slot_mapping, void* k_cache,
                                 void* v_cache, const int32_t* context_lens, const int32_t* block_tables,
                                 int64_t bt_row_stride, int32_t max_blocks, void* out, int64_t out_row_stride,
                                 int32_t batch, int32_t num_q_heads, int32_t num_kv_heads, int32_t head_dim, float scale,
                                 int64_t num_blocks, void* workspace, int64_t workspace_bytes, void* stream) {
  return nvllm::decode_common("decode_step", q, q_row_stride, key, key_row_stride, value, value_row_stride, slot_mapping,
                              k_cache, v_cache, context_lens, block_tables, bt_row_stride, max_blocks, out, out_row_stride,
                              batch, num_q_heads, num_kv_heads, head_dim, scale, num_blocks, workspace, workspace_bytes,
                              stream, true, false);
}

extern "C" int nvllm_attention_decode(const void* q, int64_t q_row_stride, const void* key, int64_t key_row_stride,
                                      const void* value, int64_t value_row_stride, const int32_t* slot_mapping, int64_t n_new,
                                      void* k_cache, void* v_cache, const int32_t* context_lens, const int32_t* block_tables,
                                      int64_t bt_row_stride, int32_t max_blocks, void* out, int64_t out_row_stride,
                                      int32_t batch, int32_t num_q_heads, int32_t num_kv_heads, int32_t head_dim, float scale,
                                      int64_t num_blocks, void* workspace, int64_t workspace_bytes, void* stream) {
  using namespace nvllm;
  // Few sequences: one launch, in which a block that meets a slot stored to takes the new row instead (one
  // sequence of 317 tokens 9.3 -> 7.0 us, eight of 100 to 1024 11.1 -> 10.0); a lane holds a slot, hence
  // the 32.  More: the copy first, under which the decode reads its lengths.
  const bool one_launch = n_new > 0 && n_new <= 32 && batch > 0 && batch <= 32;
  const int rc = store_kvcache(!one_launch, key, key_row_stride, value, value_row_stride, k_cache, v_cache, slot_mapping, n_new,
                               num_kv_heads * head_dim, num_blocks * kBlockSize, stream);
  if (rc) return rc;
  return decode_common("attention_decode", q, q_row_stride, key, key_row_stride, value, value_row_stride, slot_mapping, k_cache,
                       v_cache, context_lens, block_tables, bt_row_stride, max_blocks, out, out_row_stride, batch, num_q_heads,
                       num_kv_heads, head_dim, scale, num_blocks, workspace, workspace_bytes, stream, one_launch,
                       n_new > 0 && !one_launch, one_launch ? static_cast<int>(n_new) : 0);
}

// ---- decode without a caller-provided workspace ---------------------------------------------
//
// nvllm_decode_paged_static is for hosts that have no way to hand the library a scratch
// buffer: an engine that has already given all free HBM to its KV cache (nano-vllm sizes the
// cache from whatever memory is left, so a later allocation can fail), a real-time serving
// loop in which cudaMalloc's implicit device synchronisation is unacceptable, or a binding
// from a language that owns no device allocator and only forwards the pointers it was given.
// The arrival counters and the partials live in a fixed array that is part of the library image.

namespace nvllm {

constexpr int64_t kStaticScratchBytes = NVLLM_DECODE_STATIC_SCRATCH_BYTES;

// Lives in every context that loads this library, for the life of the process.  In host
// code this name is only a handle for cudaGetSymbolAddress, never a device address.  Like any
// file-scope device array without an initialiser it starts as zeros, which is what the
// arrival counters at its head need.
static __device__ __align__(256) unsigned char g_decode_static_scratch[kStaticScratchBytes];

// Device address of the array on each device, resolved on that device's first call.
static void* g_static_scratch_addr[64] = {nullptr};

static int static_scratch(void** out) {
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= 64) {
    (void)cudaGetLastError();
    return fail(NVLLM_E_NO_DEVICE, "decode_paged_static: no usable CUDA device is current");
  }
  if (!g_static_scratch_addr[dev]) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_decode_static_scratch);
    if (e != cudaSuccess || !p) {
      (void)cudaGetLastError();
      return fail(NVLLM_E_CUDA, "decode_paged_static: cudaGetSymbolAddress failed on device %d: %s", dev,
                  cudaGetErrorString(e));
    }
    g_static_scratch_addr[dev] = p;
  }
  *out = g_static_scratch_addr[dev];
  return NVLLM_OK;
}

cudaError_t clear_static_scratch() {
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= 64 || !g_static_scratch_addr[dev]) return e;  // not in use on this device
  e = cudaMemset(g_static_scratch_addr[dev], 0, kStaticScratchBytes);
  return e == cudaSuccess ? cudaDeviceSynchronize() : e;
}

}  // namespace nvllm

extern "C" int nvllm_decode_paged_static(const void* q, int64_t q_row_stride, const void* k_cache,
                                         const void* v_cache, const int32_t* context_lens,
                                         const int32_t* block_tables, int64_t bt_row_stride, int32_t max_blocks,
                                         void* out, int64_t out_row_stride, int32_t batch, int32_t num_q_heads,
                                         int32_t num_kv_heads, int32_t head_dim, float scale, int64_t num_blocks,
                                         void* stream) {
  using namespace nvllm;
  const int64_t need = nvllm_decode_workspace_bytes(batch, max_blocks, num_q_heads, num_kv_heads, head_dim);
  if (need < 0) return static_cast<int>(need);  // geometry rejected; message already set
  if (batch == 0) return NVLLM_OK;
  if (need > kStaticScratchBytes)
    return fail(NVLLM_E_WORKSPACE,
                "decode_paged_static: this geometry needs %lld bytes of split-KV scratch but the built-in array "
                "holds %lld; use nvllm_decode_paged with a caller-owned workspace",
                (long long)need, (long long)kStaticScratchBytes);
  void* scratch = nullptr;
  int rc = static_scratch(&scratch);
  if (rc) return rc;
  // What must start at zero are the arrival counters at the head of the array.  They are zero
  // when the library is loaded, and the block that merges a sequence's partials puts its
  // counter back to zero, so every completed call leaves them cleared for the next one.  The
  // partials themselves are always written before they are read within one call, and the marks of those that
  // are marked cells are taken off by the block that reads them.
  return nvllm_decode_paged(q, q_row_stride, k_cache, v_cache, context_lens, block_tables, bt_row_stride, max_blocks,
                            out, out_row_stride, batch, num_q_heads, num_kv_heads, head_dim, scale, num_blocks,
                            scratch, kStaticScratchBytes, stream);
}
