// Varlen causal GQA prefill, two query tiles per thread block: the large-batch form of
// prefill_tcp.cu (same math, same arguments, same item queue; nanovllm/layers/attention.py:67-73).
//
// One block per SM works on a pair of neighbouring 128-row query tiles that share every K/V tile.
// What bounds the one-tile kernel is the operand traffic of its products: with 64-key tiles an
// S product (M128 N64) reads 6 KB of shared memory per 32 cycles of arithmetic and every K/V tile is
// fetched for 128 rows only.  Here tiles are 128 keys wide (M128 N128 K16: 8 KB per 64 cycles), a K/V
// tile is loaded once for 256 rows, and while the softmax warps of one tile work, the tensor core
// has the other tile's products to do, so S needs no second buffer: 512 TMEM columns hold S (with P
// over it) and O of both tiles.
//
// Sixteen warps: 0-3 and 4-7 softmax of tile 0 and 1 (thread = query row), 8-11 epilogue of both,
// 12 TMA producer, 13 MMA issuer (one lane each), two idle; registers are handed over with
// setmaxnreg (192 / 64 / 64 per thread).  Order of the products: per key tile and query tile P V of
// that tile, then at once its next S, so that one commit per query tile and step tells the softmax
// warps that S is there, the softmax warps that O is settled (for the rare rescale), and the
// producer that a K and a V buffer are free.  The last P V of an item is followed by the first S of
// the next item.  A key tile of which at most 64 keys are visible to a query tile (diagonal,
// ragged end) is done at half width.
//
// Items (sequence, pair of query tiles, head group), head packing, the order of the items and the
// epilogue are those of prefill_tcp.cu.
#include <atomic>
#include <type_traits>

#include "common.cuh"
#include "prefill.cuh"
#include "prefill_tc.cuh"
#include "sm100.cuh"

#ifndef NVLLM_PAIR_POLY
#define NVLLM_PAIR_POLY 2
#endif

namespace nvllm {
using namespace sm100;

namespace pair {
constexpr int BM = 128, BN = 128, HALF = 64;
constexpr int NTHREADS = 512;
constexpr int REGS_SOFTMAX = 192, REGS_EPILOGUE = 64, REGS_OTHER = 64;
static_assert(256 * REGS_SOFTMAX + 128 * REGS_EPILOGUE + 128 * REGS_OTHER <= NTHREADS * 128, "register pool of a block");
constexpr int TMEM_COLS = 512;
constexpr int MAX_BATCH = kPrefillMaxBatch;
constexpr int SORT_BATCH = 512;  // batches up to this size are ranked by length
// [i]: query tile; [i][c & 1]: the c-th event of its kind for that tile.  Two barriers in turn
// where a waiter may be one event behind.
enum Bar {
  ITEM_FULL = 0, ITEM_FREE = 2, Q_FULL = 4, K_FULL = 6, V_FULL = 8, S_FULL = 10, O_FULL = 14, P_LO = 18, P_HI = 20,
  O_FREE = 22, EPI_FULL = 24, DRAIN = 28, NUM_BARS
};
template <int D_>
struct Geo {
  static constexpr int D = D_;
  static constexpr int NSUB = D / 64;  // 64-element (128-byte) sub-tiles of a row, the unit of the swizzle
  static constexpr int Q_SUB = BM * 128, Q_BYTES = NSUB * Q_SUB;
  static constexpr int KV_SUB = BN * 128, KV_BYTES = NSUB * KV_SUB;
  static constexpr int OFF_Q = 0, OFF_K = 2 * Q_BYTES, OFF_V = OFF_K + 2 * KV_BYTES;
  static constexpr int OFF_STAGE = OFF_V + 2 * KV_BYTES;  // 4 warps x 32 rows x 64 B of output
  static constexpr int OFF_CTRL = OFF_STAGE + 4 * 2048;   // barriers (8 B each)
  static constexpr int OFF_SLOTS = OFF_CTRL + 256;        // two item descriptors of 16 ints
  static constexpr int OFF_MISC = OFF_SLOTS + 128;        // tmem address, abort flag
  static constexpr int OFF_INV = OFF_MISC + 64;           // [tile][2] x 128 rows: 1 / row sum
  static constexpr int OFF_PREFIX = OFF_INV + 4 * 128 * 4;                // (MAX_BATCH + 1) ints
  static constexpr int OFF_ORDER = OFF_PREFIX + (MAX_BATCH + 1) * 4 + 4;  // MAX_BATCH u16: sequences, longest first
  static constexpr int SMEM = OFF_ORDER + MAX_BATCH * 2 + 1024;
};
static_assert(NUM_BARS * 8 <= 256, "barrier area");
static_assert(Geo<128>::SMEM <= 227 * 1024, "shared memory of an SM");
constexpr int NUM_SLOTS = 64;  // launches that may be in flight at once

struct Item {
  int b, h, m0, q0, Lq, k0, Lk;
  int n[2];   // key tiles of each query tile; n[0] < 0: no more work
  int half;   // bit i: tile i's last key tile has at most 64 visible keys
};

// 2^x for a pair, x in [-126, 127], without the special-function unit: 2^round(x) by exponent
// arithmetic, 2^f on [-1/2, 1/2] by a polynomial of degree 4 (relative error below 3e-6, a
// hundredth of what the rounding of P to bf16 leaves).
__device__ __forceinline__ void exp2_poly2(float x0, float x1, float& y0, float& y1) {
  const uint64_t magic = pack2(12582912.f, 12582912.f), nmagic = pack2(-12582912.f, -12582912.f);
  const uint64_t x = pack2(fmaxf(x0, -126.f), fmaxf(x1, -126.f));
  const uint64_t t = add2(x, magic);                      // round(x) in the low mantissa bits
  const uint64_t n = add2(t, nmagic);
  const uint64_t f = fma2(n, pack2(-1.f, -1.f), x);
  constexpr float C0 = 0.9999993f, C1 = 0.6931218f, C2 = 0.24024744f, C3 = 0.05591786f, C4 = 0.0095701f;
  uint64_t p = pack2(C4, C4);
  p = fma2(p, f, pack2(C3, C3));
  p = fma2(p, f, pack2(C2, C2));
  p = fma2(p, f, pack2(C1, C1));
  p = fma2(p, f, pack2(C0, C0));
  float p0, p1, t0, t1;
  unpack2(p, p0, p1);
  unpack2(t, t0, t1);
  y0 = __int_as_float(__float_as_int(p0) + (__float_as_int(t0) << 23));
  y1 = __int_as_float(__float_as_int(p1) + (__float_as_int(t1) << 23));
}
}  // namespace pair

// Work counters, one pair per launch slot; the last block of a launch to leave resets its pair.
__device__ unsigned int g_pair_item_counter[pair::NUM_SLOTS];
__device__ unsigned int g_pair_done_counter[pair::NUM_SLOTS];

template <int D>
__global__ void __launch_bounds__(pair::NTHREADS, 1)
prefill_pair_kernel(const PrefillParams p, const __grid_constant__ CUtensorMap tmap_q,
                    const __grid_constant__ CUtensorMap tmap_k, const __grid_constant__ CUtensorMap tmap_v,
                    const int counter_slot) {
  using namespace pair;
  using G = Geo<D>;
  constexpr int OCH = D / 32, PIECES = D / 8;
  extern __shared__ unsigned char smem_raw[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  unsigned char* base_ptr = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t bars = base + G::OFF_CTRL;
  auto bar = [&](int i) { return bars + 8u * i; };
  volatile int* slots = reinterpret_cast<volatile int*>(base_ptr + G::OFF_SLOTS);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(base_ptr + G::OFF_MISC);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(base_ptr + G::OFF_MISC + 8);
  int* prefix = reinterpret_cast<int*>(base_ptr + G::OFF_PREFIX);  // prefix[i] = items (per head group) before the i-th sequence
  unsigned short* order = reinterpret_cast<unsigned short*>(base_ptr + G::OFF_ORDER);  // order[i] = i-th longest sequence
  float* inv_buf = reinterpret_cast<float*>(base_ptr + G::OFF_INV);
  // The rows of a tile are BMT = 128 / n query tokens x n query heads of one KV head (row = token * n +
  // head); an item covers p.tiles (1 or 2) neighbouring tiles.
  const int pack = p.pack, BMT = BM / pack, IT = BMT * p.tiles;

  pdl_trigger();
  if (!p.lengths_early) pdl_wait();
  // Rank the sequences by key length, longest first (ties by index): rank = how many come before.
  if (p.batch <= SORT_BATCH) {
    const int mine = tid < p.batch ? p.cu_k[tid + 1] - p.cu_k[tid] : 0;
    if (tid < p.batch) prefix[tid] = mine;  // lengths, for a moment
    __syncthreads();
    int rank = 0;
    if (tid < p.batch)
      for (int o = 0; o < p.batch; ++o) {
        const int theirs = prefix[o];
        rank += (theirs > mine) || (theirs == mine && o < tid);
      }
    if (tid < p.batch) order[rank] = static_cast<unsigned short>(tid);
  } else {
    for (int b = tid; b < p.batch; b += NTHREADS) order[b] = static_cast<unsigned short>(b);
  }
  __syncthreads();
  if (warp == 12) {
    // items per sequence, in that order -> exclusive prefix sum (warp scan, 32 at a time)
    int carry = 0;
    for (int i0 = 0; i0 < p.batch; i0 += 32) {
      const int i = i0 + lane;
      int items = 0;
      if (i < p.batch) {
        const int b = order[i];
        items = (p.cu_q[b + 1] - p.cu_q[b] + IT - 1) / IT;
      }
      int incl = items;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += v;
      }
      if (i < p.batch) prefix[i] = carry + incl - items;
      carry += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) {
      prefix[p.batch] = carry;
      for (int i = 0; i < NUM_BARS; ++i) {
        // four softmax warps fill P and the normalisers, four epilogue warps free O; an item slot is free
        // when eight softmax warps, four epilogue warps and the MMA issuer are done with it
        const uint32_t count = (i >= P_LO && i < DRAIN) ? 4u : (i == ITEM_FREE || i == ITEM_FREE + 1) ? 13u : 1u;
        mbar_init(bar(i), count);
      }
      *abort_flag = 0;
      mbar_fence_init();
      prefetch_tmap(&tmap_q);
      prefetch_tmap(&tmap_k);
      prefetch_tmap(&tmap_v);
    }
  }
  if (warp == 13) tmem_alloc(smem_u32(tmem_slot), TMEM_COLS);
  if (p.lengths_early) pdl_wait();  // from here on q, k and v are read
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;  // S of tile i at i * 128 (P over it), O of tile i at 256 + i * 128

  auto read_item = [&](int it) {
    volatile int* s = slots + (it & 1) * 16;
    Item x;
    x.b = s[0]; x.h = s[1]; x.m0 = s[2]; x.q0 = s[3]; x.Lq = s[4]; x.k0 = s[5]; x.Lk = s[6];
    x.n[0] = s[7]; x.n[1] = s[8]; x.half = s[9];
    return x;
  };
  auto wait = [&](int b, int count) { return wait_or_abort(bar(b), count & 1, abort_flag); };
  // the c-th event of one of a tile's pairs of barriers
  auto wait2 = [&](int b, int i, int c) { return wait_or_abort(bar(b + 2 * i + (c & 1)), (c >> 1) & 1, abort_flag); };

  // The register hand-over sits inside each group's own branch: the allocator bounds the code that
  // follows a setmaxnreg on its path, and paths that merged again would all get the smallest bound.
  if (warp >= 12) {
   asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REGS_OTHER));
   if (warp == 12 && elect_one()) {
    // ------------------------------------------------------------------ producer lane
    const int hgroups = p.hq / pack;
    const int total_items = prefix[p.batch] * hgroups;
    auto decode_item = [&](unsigned idx) {
      Item x;
      while (true) {
        x.n[0] = -1;
        x.n[1] = 0;
        if (idx >= static_cast<unsigned>(total_items)) break;
        const int pi = idx / hgroups;
        x.h = (idx - pi * hgroups) * pack;  // first of the packed heads; head groups fastest: neighbours share K/V in L2
        int lo = 0, hi = p.batch;           // largest i with prefix[i] <= pi
        while (hi - lo > 1) {
          const int mid = (lo + hi) >> 1;
          if (prefix[mid] <= pi) lo = mid; else hi = mid;
        }
        x.b = order[lo];
        x.q0 = p.cu_q[x.b];
        x.Lq = p.cu_q[x.b + 1] - x.q0;
        x.k0 = p.cu_k[x.b];
        x.Lk = p.cu_k[x.b + 1] - x.k0;
        const int items = prefix[lo + 1] - prefix[lo];
        x.m0 = (items - 1 - (pi - prefix[lo])) * IT;  // a sequence's long items first
        x.half = 0;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int m = x.m0 + i * BMT;
          x.n[i] = 0;
          if (i >= p.tiles || m >= x.Lq) continue;
          const int kv_end = min(x.Lk, min(m + BMT, x.Lq) + (x.Lk - x.Lq));
          if (kv_end > 0) {
            const int halves = (kv_end + HALF - 1) / HALF;
            x.n[i] = (halves + 1) / 2;
            x.half |= (halves & 1) << i;
            continue;
          }
          // No visible key for the whole tile (only possible when Lk < Lq, which the engine never
          // produces): the rows are zero; written here, the other roles never see it.
          for (int r = m; r < min(m + BMT, x.Lq); ++r) {
            uint4* dst = reinterpret_cast<uint4*>(p.out + static_cast<int64_t>(x.q0 + r) * p.out_stride + x.h * D);
            for (int c = 0; c < PIECES * pack; ++c) dst[c] = make_uint4(0, 0, 0, 0);  // the packed heads are adjacent
          }
        }
        if (x.n[0] + x.n[1] > 0) break;
        idx = atomicAdd(&g_pair_item_counter[counter_slot], 1u);
      }
      return x;
    };
    // Which event frees a K or V buffer: the count of a tile's S (O: bit 30 set) event, tile in bit 31.
    auto event = [](int i, int count, bool o) {
      return static_cast<unsigned>(count) | (o ? 1u << 30 : 0u) | static_cast<unsigned>(i) << 31;
    };
    auto wait_event = [&](unsigned e) {
      return wait2(e >> 30 & 1u ? O_FULL : S_FULL, static_cast<int>(e >> 31), static_cast<int>(e & 0x3fffffffu));
    };
    unsigned k_free0 = 0, k_free1 = 0, v_free0 = 0, v_free1 = 0;
    int T = 0;                          // key tiles loaded so far in this block's life
    int k_loads = 0, v_loads = 0;       // K and V tiles asked for
    int s_count[2] = {0, 0};            // S events of each tile before this item
    int o_count[2] = {0, 0};            // item tiles before this item
    // The counter is read a little ahead of need (see prefill_tcp.cu).
    unsigned next_idx = atomicAdd(&g_pair_item_counter[counter_slot], 1u);
    bool ok = true;
    for (int it = 0; ok; ++it) {
      const Item x = decode_item(next_idx);
      if (it >= 2 && !wait(ITEM_FREE + (it & 1), (it >> 1) - 1)) break;
      volatile int* s = slots + (it & 1) * 16;
      s[0] = x.b; s[1] = x.h; s[2] = x.m0; s[3] = x.q0; s[4] = x.Lq; s[5] = x.k0; s[6] = x.Lk;
      s[7] = x.n[0]; s[8] = x.n[1]; s[9] = x.half;
      mbar_arrive(bar(ITEM_FULL + (it & 1)));
      if (x.n[0] < 0) break;

      const int kvh = x.h / p.g;
      const int n = max(x.n[0], x.n[1]);
      // rows of the item's last key tile: half a tile where no query tile needs more
      const bool last_half = (x.n[0] < n || (x.half & 1)) && (x.n[1] < n || (x.half & 2));
      const int32_t* bt_row = p.block_tables ? p.block_tables + x.b * p.bt_stride : nullptr;
      auto load_tile = [&](const CUtensorMap* map, int off, int full, int j, int row) {
        const int halves = j == n - 1 && last_half ? 1 : 2;
        mbar_expect_tx(bar(full), halves * (G::KV_BYTES / 2));
        for (int hh = 0; hh < halves; ++hh)
#pragma unroll
          for (int sub = 0; sub < G::NSUB; ++sub)
            tma_load_3d(base + off + sub * G::KV_SUB + hh * (HALF * 128), map, bar(full), sub * 64, kvh, row + hh * HALF);
      };
      for (int j = 0; j < n; ++j) {
        if (j == max(0, n - 2)) next_idx = atomicAdd(&g_pair_item_counter[counter_slot], 1u);
        const int t = T + j, st = t & 1;
        int row;
        if (bt_row) {
          int64_t blk = bt_row[(j * BN) / kBlockSize];
          if (blk < 0 || blk >= p.num_blocks) {
            atomicOr(p.status, NVLLM_STATUS_BAD_BLOCK);
            blk = 0;
          }
          row = static_cast<int>(blk * kBlockSize + (j * BN) % kBlockSize);
        } else {
          row = x.k0 + j * BN;
        }
        if (t >= 2 && !(ok = wait_event(st ? k_free1 : k_free0))) break;
        load_tile(&tmap_k, G::OFF_K + st * G::KV_BYTES, K_FULL + st, j, row);
        ++k_loads;
        if (j == 0) {
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            if (x.n[i] == 0) continue;
            // Q buffer: free once the previous item's last S product of this tile is complete
            if (s_count[i] > 0 && !(ok = wait2(S_FULL, i, s_count[i] - 1))) break;
            mbar_expect_tx(bar(Q_FULL + i), G::NSUB * pack * BMT * 128);
#pragma unroll
            for (int sub = 0; sub < G::NSUB; ++sub)
              tma_load_3d(base + G::OFF_Q + i * G::Q_BYTES + sub * G::Q_SUB, &tmap_q, bar(Q_FULL + i), sub * 64, x.h,
                          x.q0 + x.m0 + i * BMT);
          }
          if (!ok) break;
        }
        if (t >= 2 && !(ok = wait_event(st ? v_free1 : v_free0))) break;
        load_tile(&tmap_v, G::OFF_V + st * G::KV_BYTES, V_FULL + st, j, row);
        ++v_loads;
        const int r = j < x.n[1] ? 1 : 0;  // the query tile that uses this key tile last
        const int sr = r ? s_count[1] : s_count[0], nr = r ? x.n[1] : x.n[0], orr = r ? o_count[1] : o_count[0];
        const unsigned kf = event(r, sr + j, false), vf = j + 1 < nr ? event(r, sr + j + 1, false) : event(r, orr, true);
        if (st) {
          k_free1 = kf;
          v_free1 = vf;
        } else {
          k_free0 = kf;
          v_free0 = vf;
        }
      }
      T += n;
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        s_count[i] += x.n[i];
        o_count[i] += x.n[i] > 0;
      }
    }
    if (*abort_flag) {  // no copy may land after the block has left
      for (int back = 1; back <= 2; ++back) {
        if (k_loads >= back) (void)mbar_wait(bar(K_FULL + ((k_loads - back) & 1)), ((k_loads - back) >> 1) & 1);
        if (v_loads >= back) (void)mbar_wait(bar(V_FULL + ((v_loads - back) & 1)), ((v_loads - back) >> 1) & 1);
      }
    }
   } else if (warp == 13 && elect_one()) {
    // ------------------------------------------------------------------ MMA issuer
    const uint64_t q_desc = umma_desc(base + G::OFF_Q, 16, 1024);
    const uint64_t k_desc = umma_desc(base + G::OFF_K, 16, 1024);
    const uint64_t v_desc = umma_desc(base + G::OFF_V, G::KV_SUB, 1024);
    constexpr uint32_t idesc_pv = umma_idesc(BM, D, 0, 1);
    int s_count[2] = {0, 0}, o_count[2] = {0, 0}, lo_count[2] = {0, 0}, hi_count[2] = {0, 0};
    auto last_half = [](const Item& x, int i, int j) { return j == x.n[i] - 1 && (x.half >> i & 1); };
    // S of tile i and key tile t (number j of the item)
    auto issue_s = [&](const Item& x, int i, int j, int t) -> bool {
      if (j == 0 && !wait(Q_FULL + i, o_count[i])) return false;
      if (!wait(K_FULL + (t & 1), t >> 1)) return false;
      tc_fence_after();
      const uint32_t idesc = last_half(x, i, j) ? umma_idesc(BM, HALF, 0, 0) : umma_idesc(BM, BN, 0, 0);
      const uint64_t qd = q_desc + static_cast<uint64_t>(i * (G::Q_BYTES >> 4));
      const uint64_t kd = k_desc + static_cast<uint64_t>((t & 1) * (G::KV_BYTES >> 4));
#pragma unroll
      for (int ks = 0; ks < D / 16; ++ks) {
        const uint64_t qoff = ((ks >> 2) * G::Q_SUB + (ks & 3) * 32) >> 4;
        const uint64_t koff = ((ks >> 2) * G::KV_SUB + (ks & 3) * 32) >> 4;
        umma_ss(tmem + i * 128, qd + qoff, kd + koff, idesc, ks > 0);
      }
      umma_commit(bar(S_FULL + 2 * i + (s_count[i] & 1)));
      ++s_count[i];
      return true;
    };
    auto issue_pv = [&](const Item& x, int i, int j, int t) -> bool {
      if (!wait(V_FULL + (t & 1), t >> 1)) return false;
      // the first product of an item overwrites O: the previous item's O must have been read
      if (j == 0 && o_count[i] > 0 && !wait(O_FREE + i, o_count[i] - 1)) return false;
      const uint64_t vd = v_desc + static_cast<uint64_t>((t & 1) * (G::KV_BYTES >> 4));
      const int halves = last_half(x, i, j) ? 1 : 2;
      for (int hh = 0; hh < halves; ++hh) {
        if (!(hh == 0 ? wait(P_LO + i, lo_count[i]++) : wait(P_HI + i, hi_count[i]++))) return false;
        tc_fence_after();
#pragma unroll
        for (int ks = 0; ks < HALF / 16; ++ks)
          umma_ts(tmem + 256 + i * 128, tmem + i * 128 + hh * 32 + ks * 8,
                  vd + static_cast<uint64_t>(((hh * 4 + ks) * 2048) >> 4), idesc_pv, (j > 0 || hh > 0 || ks > 0) ? 1u : 0u);
      }
      return true;
    };
    int T = 0;
    bool ok = wait(ITEM_FULL, 0);
    Item x;
    x.n[0] = -1;
    if (ok) x = read_item(0);
    if (ok && x.n[0] >= 0) {
#pragma unroll
      for (int i = 0; i < 2; ++i)
        if (ok && x.n[i] > 0) ok = issue_s(x, i, 0, 0);
    }
    for (int it = 0; ok && x.n[0] >= 0; ++it) {
      const int n = max(x.n[0], x.n[1]);
      Item y;
      y.n[0] = y.n[1] = -1;
      bool have_next = false;
      int begun = 0;  // tiles whose first S of the next item has been issued
      for (int j = 0; ok && j < n; ++j) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          if (!ok || j >= x.n[i]) continue;
          if (!(ok = issue_pv(x, i, j, T + j))) break;
          if (j + 1 < x.n[i]) {
            ok = issue_s(x, i, j + 1, T + j + 1);
            continue;
          }
          umma_commit(bar(O_FULL + 2 * i + (o_count[i] & 1)));
          ++o_count[i];
          if (!have_next) {
            if (!(ok = wait(ITEM_FULL + ((it + 1) & 1), (it + 1) >> 1))) break;
            y = read_item(it + 1);
            have_next = true;
          }
          // first S of the next item, tile 0's always before tile 1's (the producer counts on it)
          if (y.n[i] > 0 && (i == 0 || y.n[0] == 0 || (begun & 1))) {
            ok = issue_s(y, i, 0, T + n);
            begun |= 1 << i;
          }
        }
      }
      if (!ok) break;
#pragma unroll
      for (int i = 0; i < 2; ++i)
        if (ok && y.n[i] > 0 && !(begun >> i & 1)) ok = issue_s(y, i, 0, T + n);
      T += n;
      mbar_arrive(bar(ITEM_FREE + (it & 1)));
      x = y;
    }
    if (!ok) {  // make sure nothing is still running on TMEM before it is freed
      umma_commit(bar(DRAIN));
      (void)mbar_wait(bar(DRAIN), 0);
    }
   }
  } else if (warp < 8) {
    // ------------------------------------------------------------------ softmax rows
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(REGS_SOFTMAX));
    const int i = warp >> 2, r = (warp & 3) * 32 + lane;  // query tile, row
    const int r_tok = r / pack;  // this row's token within the tile (== BMT for the unused rows of a 7-head tile)
    const uint32_t lane_addr = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t tmem_s = tmem + i * 128 + lane_addr, tmem_o = tmem + 256 + i * 128 + lane_addr;
    const uint64_t scale2 = pack2(p.scale_log2e, p.scale_log2e);
    int s_count = 0, o_count = 0, T = 0;
    float m_used = -INFINITY, l = 0.f;
    bool ok = true;

    // One key tile: NC visible columns at most, `limit` the last visible one.
    auto key_tile = [&](auto width, auto masked, int limit, int j, int t, int dead) -> bool {
      constexpr int NC = decltype(width)::value;
      constexpr bool MASKED = decltype(masked)::value;
      uint32_t s[NC];
#pragma unroll
      for (int c = 0; c < NC / 32; ++c) tmem_ld32(tmem_s + c * 32, *reinterpret_cast<uint32_t(*)[32]>(&s[c * 32]));
      tmem_wait_ld();
      if constexpr (MASKED) {
#pragma unroll
        for (int c = 0; c < NC; ++c)
          if (c > limit) s[c] = 0xff800000u;  // -inf
      }
      float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int c = 0; c < NC; c += 8) {
#pragma unroll
        for (int k = 0; k < 4; ++k)
          mx4[k] = fmax3(mx4[k], __uint_as_float(s[c + 2 * k]), __uint_as_float(s[c + 2 * k + 1]));
      }
      const float mx = fmax3(fmaxf(mx4[0], mx4[1]), mx4[2], mx4[3]);
      const float m_new = fmaxf(m_used, mx * p.scale_log2e);
      // lazy rescale: keep the old reference maximum unless it has been outgrown by 2^8
      const bool grow = m_new > m_used + tc::kRescaleThreshold;
      if (__any_sync(0xffffffffu, grow)) {
        float alpha = 1.f;
        if (grow) {
          alpha = (m_used == -INFINITY) ? 0.f : fast_exp2(m_used - m_new);
          m_used = m_new;
          l *= alpha;
        }
        if (j > 0) {  // O holds tiles 0..j-1: their products were issued before this S, which is complete
#pragma unroll 1
          for (int c = 0; c < D / 16; ++c) {
            uint32_t o[16];
            tmem_ld16(tmem_o + c * 16, o);
            tmem_wait_ld();
#pragma unroll
            for (int e = 0; e < 16; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * alpha);
            tmem_st16(tmem_o + c * 16, o);
          }
        }
      }
      if (dead < NC) {
        // Last tile of the sequence: V rows past the end hold whatever the cache block (or the next
        // sequence) has there.  Their P is 0, but 0 x NaN would still poison O, so the rows are cleared
        // in shared memory before the product is issued (by both query tiles where both use them).
        if (!wait(V_FULL + (t & 1), t >> 1)) return false;
        unsigned char* vt = base_ptr + G::OFF_V + (t & 1) * G::KV_BYTES;
        for (int k = r; k < (NC - dead) * PIECES; k += 128) {
          const int row = dead + k / PIECES, piece = k % PIECES;
          *reinterpret_cast<uint4*>(vt + (piece >> 3) * G::KV_SUB + row * 128 + (piece & 7) * 16) = make_uint4(0, 0, 0, 0);
        }
        fence_proxy_async();
      }
      const float msub = (m_used == -INFINITY) ? 0.f : m_used;
      // p = 2^(s * scale - m): the multiply-subtract and the row sum run two lanes at a time; P is packed
      // in place, s[c] <- (p[2c], p[2c+1]), and handed over in halves so that the product can start
      const uint64_t nmsub2 = pack2(-msub, -msub);
      uint64_t sum2[2] = {0ull, 0ull};
#pragma unroll
      for (int hh = 0; hh < NC / HALF; ++hh) {
#pragma unroll
        for (int c = hh * 32; c < hh * 32 + 32; ++c) {
          float a0, a1, p0, p1;
          unpack2(fma2(pack2(__uint_as_float(s[2 * c]), __uint_as_float(s[2 * c + 1])), scale2, nmsub2), a0, a1);
          if (!MASKED && c % 8 < NVLLM_PAIR_POLY) {
            exp2_poly2(a0, a1, p0, p1);
          } else {
            p0 = fast_exp2(a0);
            p1 = fast_exp2(a1);
          }
          sum2[c & 1] = add2(sum2[c & 1], pack2(p0, p1));
          s[c] = pack_bf16x2(p0, p1);
        }
        tmem_st32(tmem_s + hh * 32, *reinterpret_cast<uint32_t(*)[32]>(&s[hh * 32]));
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar((hh == 0 ? P_LO : P_HI) + i));
      }
      float t0, t1, t2, t3;
      unpack2(sum2[0], t0, t1);
      unpack2(sum2[1], t2, t3);
      l += (t0 + t1) + (t2 + t3);
      return true;
    };

    for (int it = 0; ok; ++it) {
      if (!(ok = wait(ITEM_FULL + (it & 1), it >> 1))) break;
      const Item x = read_item(it);
      if (x.n[0] < 0) break;
      const int n = i ? x.n[1] : x.n[0];
      const int m0 = x.m0 + i * BMT, off = x.Lk - x.Lq, last_key = min(m0 + r_tok + off, x.Lk - 1);
      m_used = -INFINITY;
      l = 0.f;
      for (int j = 0; j < n; ++j) {
        if (!(ok = wait2(S_FULL, i, s_count))) break;
        ++s_count;
        tc_fence_after();
        const int j0 = j * BN, limit = last_key - j0, dead = x.Lk - j0;
        const bool half = j == n - 1 && (x.half >> i & 1);
        const int nc = half ? HALF : BN;
        const bool masked = j0 + nc - 1 > m0 + off || nc > dead;  // touches the diagonal or the end
        using W = std::integral_constant<int, BN>;
        using H = std::integral_constant<int, HALF>;
        if (!half) ok = masked ? key_tile(W{}, std::true_type{}, limit, j, T + j, dead) : key_tile(W{}, std::false_type{}, limit, j, T + j, dead);
        else ok = key_tile(H{}, std::true_type{}, limit, j, T + j, dead);
        if (!ok) break;
      }
      if (!ok) break;
      T += max(x.n[0], x.n[1]);
      if (n > 0) {  // the row's normaliser goes to the epilogue warps; this warp is done with the item
        inv_buf[(i * 2 + (o_count & 1)) * 128 + r] = l > 0.f ? 1.f / l : 0.f;
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(EPI_FULL + 2 * i + (o_count & 1)));
        ++o_count;
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(ITEM_FREE + (it & 1)));
    }
  } else {
    // ------------------------------------------------------------------ epilogue rows
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REGS_EPILOGUE));
    const int ew = warp & 3, r = ew * 32 + lane;
    const uint32_t lane_addr = static_cast<uint32_t>(ew * 32) << 16;
    unsigned char* stage = base_ptr + G::OFF_STAGE + ew * 2048;  // this warp's 32 rows x 64 B
    int o_count[2] = {0, 0};
    bool ok = true;
    for (int it = 0; ok; ++it) {
      if (!(ok = wait(ITEM_FULL + (it & 1), it >> 1))) break;
      const Item x = read_item(it);
      if (x.n[0] < 0) break;
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        if (x.n[i] == 0) continue;
        const int oc = o_count[i]++;
        if (!(ok = wait2(EPI_FULL, i, oc))) break;
        const float inv = inv_buf[(i * 2 + (oc & 1)) * 128 + r];
        if (!(ok = wait2(O_FULL, i, oc))) break;
        tc_fence_after();
        // epilogue: O / l -> bf16; 32 columns at a time through this warp's patch of shared memory
        const int srow = lane >> 2, spiece = lane & 3;  // the eight 64-byte row segments one store instruction writes
        const int m0 = x.m0 + i * BMT;
        __nv_bfloat16* out_tile = p.out + static_cast<int64_t>(x.q0 + m0) * p.out_stride + x.h * D;
        const int toks_valid = min(BMT, x.Lq - m0);
#pragma unroll
        for (int c = 0; c < OCH; ++c) {
          uint32_t o[32];
          tmem_ld32(tmem + 256 + i * 128 + lane_addr + c * 32, o);
          tmem_wait_ld();
          if (c == OCH - 1) {  // O is in registers: the next item's first product may overwrite it
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(O_FREE + i));
          }
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            uint32_t w[4];
#pragma unroll
            for (int e = 0; e < 4; ++e)
              w[e] = pack_bf16x2(__uint_as_float(o[8 * k + 2 * e]) * inv, __uint_as_float(o[8 * k + 2 * e + 1]) * inv);
            *reinterpret_cast<uint4*>(stage + lane * 64 + ((k ^ ((lane >> 1) & 3)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
          }
          __syncwarp();
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const int lr = k * 8 + srow;       // row within the warp's 32
            const int row = ew * 32 + lr;      // row of the tile
            const int tok = row / pack, hh = row - tok * pack;
            const uint4 v = *reinterpret_cast<const uint4*>(stage + lr * 64 + ((spiece ^ ((lr >> 1) & 3)) << 4));
            if (tok < toks_valid)
              *reinterpret_cast<uint4*>(out_tile + static_cast<int64_t>(tok) * p.out_stride + hh * D + c * 32 + spiece * 8) = v;
          }
          __syncwarp();
        }
      }
      if (!ok) break;
      if (lane == 0) mbar_arrive(bar(ITEM_FREE + (it & 1)));
    }
  }

  tc_fence_before();
  __syncthreads();
  if (tid == 0) {
    if (*abort_flag) atomicOr(p.status, NVLLM_STATUS_TIMEOUT);
    // the last block to leave re-arms this launch slot's counters
    if (atomicAdd(&g_pair_done_counter[counter_slot], 1u) == gridDim.x - 1) {
      g_pair_item_counter[counter_slot] = 0;
      g_pair_done_counter[counter_slot] = 0;
      __threadfence();
    }
  }
  if (warp == 13) {
    tc_fence_after();
    tmem_dealloc(tmem, TMEM_COLS);
  }
}

// ---- host side ---------------------------------------------------------------------------

template <int D>
static int launch_prefill_pair_t(const PrefillParams& p, const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv,
                                 int64_t max_items, cudaStream_t stream) {
  using G = pair::Geo<D>;
  static bool attr_done[64] = {false};
  static std::atomic<unsigned> launch_seq{0};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return fail(NVLLM_E_NO_DEVICE, "prefill: device index %d out of range", dev);
  if (!attr_done[dev]) {
    cudaError_t e = cudaFuncSetAttribute(prefill_pair_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, G::SMEM);
    // The warp groups trade registers inside the pool the block gets at launch (threads x the kernel's
    // register count); a build whose count is lower could never satisfy the softmax groups' request, and
    // that request waits without a bound.
    cudaFuncAttributes attr;
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&attr, prefill_pair_kernel<D>);
    if (e != cudaSuccess) return fail(NVLLM_E_CUDA, "prefill (pairs): set-up failed: %s", cudaGetErrorString(e));
    constexpr int need = 256 * pair::REGS_SOFTMAX + 128 * pair::REGS_EPILOGUE + 128 * pair::REGS_OTHER;
    if (attr.numRegs * pair::NTHREADS < need)
      return fail(NVLLM_E_CUDA, "prefill (pairs): built with %d registers per thread, the warp groups' hand-over needs %d", attr.numRegs,
                  (need + pair::NTHREADS - 1) / pair::NTHREADS);
    attr_done[dev] = true;
  }
  int grid = num_sms();
  if (grid <= 0) return fail(NVLLM_E_NO_DEVICE, "prefill: no CUDA device is usable");
  if (max_items < grid) grid = static_cast<int>(max_items);
  // the two head_dim instantiations share the counter array: give each its own half
  const int slot = static_cast<int>(launch_seq.fetch_add(1) % (pair::NUM_SLOTS / 2)) + (D == 64 ? pair::NUM_SLOTS / 2 : 0);
  return launch_kernel("prefill (pairs)", prefill_pair_kernel<D>, dim3(grid), dim3(pair::NTHREADS), G::SMEM, stream, p, mq, mk, mv,
                       slot);
}

int launch_prefill_pair(const PrefillParams& p, const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv,
                        int64_t max_items, cudaStream_t stream) {
  if (p.d == 128) return launch_prefill_pair_t<128>(p, mq, mk, mv, max_items, stream);
  return launch_prefill_pair_t<64>(p, mq, mk, mv, max_items, stream);
}

}  // namespace nvllm
