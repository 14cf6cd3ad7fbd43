// Fused pre-attention step: per-head RMSNorm of q and k, NeoX-style rotary embedding of q and
// k, and the scatter of the new K/V rows into the paged cache, in one launch over the fused
// qkv activation.
//
// It stands where four launches stand in nano-vllm's Qwen3 attention block
// (nanovllm/models/qwen3.py:89-107): q_norm and k_norm (RMSNorm.rms_forward,
// nanovllm/layers/layernorm.py:17-27), rotary_emb (RotaryEmbedding.forward and
// apply_rotary_emb, nanovllm/layers/rotary_embedding.py:6-16,39-55) and store_kvcache
// (nanovllm/layers/attention.py:32-39).  Qwen2 has no q/k norm (nanovllm/models/qwen2.py:87-90):
// the weights are then NULL and only rotation and store happen.
//
// The arithmetic repeats the reference's roundings: x -> fp32, x * rsqrt(mean(x^2) + eps) rounded
// to bf16, times the bf16 weight rounded to bf16; rotation in fp32 as x1*cos - x2*sin and
// x2*cos + x1*sin with separately rounded products (no fused multiply-add), rounded to bf16.
// q and k are rewritten in place in the qkv buffer (the attention kernels read them from
// there); the rotated k row and the untouched v row are also copied to their cache slot.
//
// Bound by memory: 18 KB per token in the Qwen3-0.6B geometry.  A head is held in 16-byte pieces by D/8
// neighbouring lanes (16 for head_dim 128), so a warp works on 256 / D heads at a time; the
// rotation partner x[i +- D/2] sits D/16 lanes away and comes by shuffle, as packed bf16 (what is
// rotated has been rounded to bf16 already).  Large launches move whole token rows through shared
// memory with bulk copies: the row with its cos / sin row in, q and k back, and the K and V rows to
// their cache slots, each one copy.  16384 tokens (302 MB): 117 us with one warp per head and 4-byte
// accesses, 63 us with 16-byte accesses from registers, 57 us so.
#include <algorithm>

#include "common.cuh"
#include "sm100.cuh"

namespace nvllm {

struct PreAttnParams {
  __nv_bfloat16* qkv;
  int64_t row_stride;
  const int64_t* positions;
  const __nv_bfloat16* q_weight;  // nullable
  const __nv_bfloat16* k_weight;  // nullable
  const float* cos_sin;           // [max_position, D]: cos (D/2) then sin (D/2)
  int64_t max_position;
  float eps;
  const int32_t* slot_mapping;    // nullable: no store
  __nv_bfloat16* k_cache;
  __nv_bfloat16* v_cache;
  int64_t num_slots;
  int64_t n_tokens;
  int hq, hkv;
  bool tables_aligned;  // weights and cos / sin table start on 16-byte boundaries
  int* status;
};

// Eight bf16 as four pairs of fp32 in the packed two-lane form (sm_100 multiplies and adds those at
// one instruction per pair, rounded like the scalar ones), and back.
__device__ __forceinline__ void unpack8(const uint4& v, uint64_t (&x)[4]) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) x[i] = pack2(__uint_as_float(w[i] << 16), __uint_as_float(w[i] & 0xffff0000u));
}
__device__ __forceinline__ uint4 pack8(const uint64_t (&x)[4]) {
  uint32_t w[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float lo, hi;
    unpack2(x[i], lo, hi);
    w[i] = pack_bf16x2(lo, hi);
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}
// bf16 products rounded once, as an fp32 product (exact for two bf16) rounded to bf16 is.
__device__ __forceinline__ uint32_t mul_bf16x2(uint32_t a, uint32_t b) {
  const __nv_bfloat162 r = __hmul2_rn(*reinterpret_cast<__nv_bfloat162*>(&a), *reinterpret_cast<__nv_bfloat162*>(&b));
  return *reinterpret_cast<const uint32_t*>(&r);
}

// Eight weights / table entries of a lane; the tables need no alignment beyond their element's.
__device__ __forceinline__ uint4 load_weights(const __nv_bfloat16* w, bool aligned) {
  if (aligned) return __ldg(reinterpret_cast<const uint4*>(w));
  const unsigned short* u = reinterpret_cast<const unsigned short*>(w);
  return make_uint4(u[0] | u[1] << 16, u[2] | u[3] << 16, u[4] | u[5] << 16, u[6] | u[7] << 16);
}
__device__ __forceinline__ void load_table(const float* t, bool aligned, uint64_t (&x)[4]) {
  if (aligned) {
    const float4 a = __ldg(reinterpret_cast<const float4*>(t)), b = __ldg(reinterpret_cast<const float4*>(t) + 1);
    x[0] = pack2(a.x, a.y);
    x[1] = pack2(a.z, a.w);
    x[2] = pack2(b.x, b.y);
    x[3] = pack2(b.z, b.w);
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i) x[i] = pack2(__ldg(t + 2 * i), __ldg(t + 2 * i + 1));
  }
}

// RMSNorm (when `norm`) and rotation of one head, eight elements per lane of a group of D/8; all lanes of
// the warp call it.  c, s: the lane's cosines, and its sines with the sign of its half.
template <int D>
__device__ __forceinline__ uint4 norm_rotate(uint4 raw, bool norm, const uint4& w, float eps, const uint64_t (&c)[4],
                                             const uint64_t (&s)[4]) {
  constexpr int LANES = D / 8;
  uint64_t x[4], y[4];
  if (norm) {  // uniform over the launch
    unpack8(raw, x);
    uint64_t sq = mul2(x[0], x[0]);
#pragma unroll
    for (int i = 1; i < 4; ++i) sq = fma2(x[i], x[i], sq);
    float ss, ss1;
    unpack2(sq, ss, ss1);
    ss += ss1;
#pragma unroll
    for (int sh = LANES / 2; sh > 0; sh >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, sh);
    const float rstd = rsqrtf(ss * (1.0f / D) + eps);
#pragma unroll
    for (int i = 0; i < 4; ++i) x[i] = mul2(x[i], pack2(rstd, rstd));
    const uint4 n = pack8(x);
    raw = make_uint4(mul_bf16x2(n.x, w.x), mul_bf16x2(n.y, w.y), mul_bf16x2(n.z, w.z), mul_bf16x2(n.w, w.w));
  }
  uint4 other;
  other.x = __shfl_xor_sync(0xffffffffu, raw.x, LANES / 2);
  other.y = __shfl_xor_sync(0xffffffffu, raw.y, LANES / 2);
  other.z = __shfl_xor_sync(0xffffffffu, raw.z, LANES / 2);
  other.w = __shfl_xor_sync(0xffffffffu, raw.w, LANES / 2);
  unpack8(raw, x);
  unpack8(other, y);
#pragma unroll
  for (int i = 0; i < 4; ++i) x[i] = add2(mul2(x[i], c[i]), mul2(y[i], s[i]));
  return pack8(x);
}
// Sign of the sines: x1 cos - x2 sin in the lower half, x2 cos + x1 sin in the upper.
__device__ __forceinline__ void sign_sines(bool upper, uint64_t (&s)[4]) {
  if (upper) return;
#pragma unroll
  for (int i = 0; i < 4; ++i) s[i] ^= 0x8000000080000000ull;
}
__device__ __forceinline__ int64_t clamp_position(int64_t pos, int64_t max_position) {
  return pos < 0 ? 0 : (pos >= max_position ? max_position - 1 : pos);
}

// ---- small launches: a head per lane group ---------------------------------------------------

constexpr int kPreThreads = 256;

// AHEAD: the position is read as it stands before the previous kernel is done; the table row is then fetched by it
// together with the activation, and again if the position has changed.  From 64 tokens on, where that takes a trip to
// memory off the launch (100 tokens, 16 / 8 heads, in a chain 3.29 -> 2.85 us, 300 3.42 -> 2.96, 700 5.65 -> 5.23); with
// fewer the row is there as soon (one token 1.87 -> 1.95, 16 2.09 -> 2.10).
constexpr int64_t kAheadFromTokens = 64;

template <int D, bool AHEAD>
__global__ void __launch_bounds__(kPreThreads) pre_attention_kernel(const PreAttnParams p) {
  pdl_trigger();  // lets the attention kernel that follows get its blocks resident early
  constexpr int LANES = D / 8;  // lanes of a head
  const int sub = threadIdx.x & (LANES - 1);
  const unsigned heads = p.hq + 2 * p.hkv;
  const unsigned unit = blockIdx.x * (kPreThreads / LANES) + threadIdx.x / LANES;
  // The whole warp stays to the end (it shuffles); lane groups past the last head do nothing else.
  const bool live = unit < p.n_tokens * heads;
  const unsigned tok = live ? unit / heads : 0;
  const int head = live ? static_cast<int>(unit - tok * heads) : 0;
  uint4* row = reinterpret_cast<uint4*>(p.qkv + tok * p.row_stride + static_cast<int64_t>(head) * D) + sub;
  // The row on its way to L2 (where whatever is still written to it goes too): its trip after the wait is then one to L2
  // even while the attention kernel behind brings its first tiles there (28 captured layers of 16 sequences 380 -> 375 us,
  // 24 at 14 / 2 heads of 64 167 -> 162).  Not in front of a position that is read ahead: its trip is the one that counts
  // there (64 tokens, 14 / 2 heads of 64, in a chain 2.25 us with it, 2.02 without, 32 / 8 heads 2.65, 2.49).
  if (!AHEAD) {
    asm volatile("prefetch.global.L2 [%0];" ::"l"(row));
    pdl_wait();
  }
  int64_t guess = 0;
  if (AHEAD) {
    guess = clamp_position(__ldcg(reinterpret_cast<const long long*>(p.positions) + tok), p.max_position);  // goes round L1
    pdl_wait();
  }
  uint4 raw = *row;
  uint64_t c[4], s[4];
  auto fetch = [&](int64_t at) {
    load_table(p.cos_sin + at * D + (sub % (LANES / 2)) * 8, p.tables_aligned, c);
    load_table(p.cos_sin + at * D + D / 2 + (sub % (LANES / 2)) * 8, p.tables_aligned, s);
  };
  if (AHEAD) fetch(guess);
  const int64_t pos = clamp_position(p.positions[tok], p.max_position);
  int64_t slot = -1;
  if (p.slot_mapping && head >= p.hq) {
    slot = p.slot_mapping[tok];
    if (slot >= p.num_slots) {
      if (sub == 0 && live) atomicOr(p.status, NVLLM_STATUS_BAD_SLOT);
      slot = -1;
    }
  }
  uint4 w = make_uint4(0, 0, 0, 0);
  if (p.q_weight) w = load_weights((head < p.hq ? p.q_weight : p.k_weight) + sub * 8, p.tables_aligned);
  if (!AHEAD || pos != guess) fetch(pos);
  sign_sines(sub >= LANES / 2, s);
  const uint4 turned = norm_rotate<D>(raw, p.q_weight != nullptr, w, p.eps, c, s);
  if (!live) return;
  if (head < p.hq + p.hkv) *row = raw = turned;
  if (slot >= 0) {
    __nv_bfloat16* cache = head < p.hq + p.hkv ? p.k_cache + (slot * p.hkv + (head - p.hq)) * D
                                               : p.v_cache + (slot * p.hkv + (head - p.hq - p.hkv)) * D;
    reinterpret_cast<uint4*>(cache)[sub] = raw;
  }
}

template <int D>
static int launch_pre_attention(const PreAttnParams& p, cudaStream_t stream) {
  const int64_t units = p.n_tokens * (p.hq + 2 * p.hkv);
  constexpr int per_block = kPreThreads / (D / 8);
  if (units > 0x7fffffffLL) return fail(NVLLM_E_GEOMETRY, "qk_norm_rope_store: too many tokens for one launch");
  auto kernel = p.n_tokens >= kAheadFromTokens ? pre_attention_kernel<D, true> : pre_attention_kernel<D, false>;
  return launch_kernel("qk_norm_rope_store", kernel, dim3(static_cast<unsigned>((units + per_block - 1) / per_block)),
                       dim3(kPreThreads), 0, stream, p);
}

// ---- large launches: token rows fetched and put back by bulk copies ----------------------------------

// Stages of a ring and warps of a block: two warps are the best over rows of 2.3 to 12 KB (one: 101 us for
// 16384 rows of 12 KB instead of 74; four: 80; eight: 91), a fourth stage gives nothing.
constexpr int kRowStages = 3, kRowWarps = 2;
constexpr int64_t kRowsFromBytes = 6 << 20;  // launches from here on: see the dispatch

__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src),
               "r"(bytes), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void bulk_store(void* dst, uint32_t src, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(src), "r"(bytes) : "memory");
}

// A block works on one token at a time out of a ring of kRowStages rows (and their cos / sin rows) in
// shared memory; as many small blocks as fit keep 100 KB of loads in flight per SM without a register
// for them.
template <int D>
__global__ void __launch_bounds__(kRowWarps * 32) pre_attention_rows_kernel(const PreAttnParams p, const int stage_bytes) {
  using namespace sm100;
  pdl_prologue();
  constexpr int LANES = D / 8, GROUPS = kRowWarps * 32 / LANES, TABLE_BYTES = D * 4, HEAD_BYTES = D * 2;
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ __align__(8) uint64_t bars[kRowStages];
  __shared__ int s_slot[kRowStages];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, sub = lane & (LANES - 1), group = threadIdx.x / LANES;
  const int64_t stride = gridDim.x;
  const int n_mine = static_cast<int>((p.n_tokens - blockIdx.x + stride - 1) / stride);  // tokens blockIdx.x + k * gridDim.x
  const bool store = p.slot_mapping != nullptr;
  const int n_turn = p.hq + p.hkv;  // heads that are rotated; the V heads are only fetched to be stored
  const uint32_t turn_bytes = n_turn * HEAD_BYTES, kv_bytes = p.hkv * HEAD_BYTES;
  const uint32_t base = smem_u32(smem);
  auto bar = [&](int st) { return smem_u32(&bars[st]); };
  if (threadIdx.x == 0) {
    for (int st = 0; st < kRowStages; ++st) mbar_init(bar(st), 1);
    mbar_fence_init();
  }
  __syncthreads();

  int64_t pos_ahead = 0;
  int slot_ahead = -1;  // lane l: position and slot of the l-th token of the current 32
  auto fetch = [&](int k) {  // token k into its stage; the first warp's work
    if (k % 32 == 0 && k + lane < n_mine) {
      const int64_t tok = blockIdx.x + (k + lane) * stride;
      pos_ahead = clamp_position(p.positions[tok], p.max_position);
      if (store) slot_ahead = p.slot_mapping[tok];
    }
    const int64_t pos = __shfl_sync(0xffffffffu, pos_ahead, k % 32);
    const int slot = __shfl_sync(0xffffffffu, slot_ahead, k % 32);
    if (lane == 0) {
      const int st = k % kRowStages;
      const uint32_t dst = base + st * stage_bytes;
      s_slot[st] = slot;
      mbar_expect_tx(bar(st), turn_bytes + (store ? kv_bytes : 0) + TABLE_BYTES);
      bulk_load(dst + TABLE_BYTES, p.qkv + (blockIdx.x + k * stride) * p.row_stride, turn_bytes + (store ? kv_bytes : 0), bar(st));
      bulk_load(dst, p.cos_sin + pos * D, TABLE_BYTES, bar(st));
    }
  };
  if (warp == 0)
    for (int k = 0; k < kRowStages - 1 && k < n_mine; ++k) fetch(k);

  uint4 wq = make_uint4(0, 0, 0, 0), wk = wq;
  if (p.q_weight) {
    wq = load_weights(p.q_weight + sub * 8, true);
    wk = load_weights(p.k_weight + sub * 8, true);
  }
  bool ok = true;
  for (int i = 0; i < n_mine; ++i) {
    const int st = i % kRowStages;
    const uint32_t table = base + st * stage_bytes, row = table + TABLE_BYTES;
    // A copy never fails; bounded like every wait, after which nothing is waited for any more.
    if (ok && !(ok = mbar_wait(bar(st), (i / kRowStages) & 1))) atomicOr(p.status, NVLLM_STATUS_TIMEOUT);
    uint64_t c[4], s[4];
    const uint32_t mine = table + (sub % (LANES / 2)) * 32;
    auto pairs_of = [](const uint4& v, uint64_t& a, uint64_t& b) {
      a = pack2(__uint_as_float(v.x), __uint_as_float(v.y));
      b = pack2(__uint_as_float(v.z), __uint_as_float(v.w));
    };
    pairs_of(ld_shared16(mine), c[0], c[1]);
    pairs_of(ld_shared16(mine + 16), c[2], c[3]);
    pairs_of(ld_shared16(mine + TABLE_BYTES / 2), s[0], s[1]);
    pairs_of(ld_shared16(mine + TABLE_BYTES / 2 + 16), s[2], s[3]);
    sign_sines(sub >= LANES / 2, s);
    for (int h0 = 0; h0 < n_turn; h0 += GROUPS) {  // the same count for every lane: the rotation shuffles
      const int head = h0 + group;
      const uint32_t at = row + min(head, n_turn - 1) * HEAD_BYTES + sub * 16;
      const uint4 turned = norm_rotate<D>(ld_shared16(at), p.q_weight != nullptr, head < p.hq ? wq : wk, p.eps, c, s);
      if (head < n_turn) st_shared16(at, turned);
    }
    fence_proxy_async();
    __syncthreads();
    if (threadIdx.x == 0) {
      bulk_store(p.qkv + (blockIdx.x + i * stride) * p.row_stride, row, turn_bytes);
      const int64_t slot = s_slot[st];
      if (slot >= p.num_slots) {
        if (store) atomicOr(p.status, NVLLM_STATUS_BAD_SLOT);
      } else if (slot >= 0) {
        bulk_store(p.k_cache + slot * p.hkv * D, row + turn_bytes - kv_bytes, kv_bytes);
        bulk_store(p.v_cache + slot * p.hkv * D, row + turn_bytes, kv_bytes);
      }
      asm volatile("cp.async.bulk.commit_group;" ::: "memory");
      // the next fetch goes over token i - 1's stage: its stores must have read it
      asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
    }
    if (warp == 0) {
      __syncwarp();
      if (i + kRowStages - 1 < n_mine) fetch(i + kRowStages - 1);
    }
  }
  if (threadIdx.x == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

template <int D>
static int launch_pre_attention_rows(const PreAttnParams& p, int blocks_per_sm, int stage_bytes, int sms, cudaStream_t stream) {
  static bool attr_set[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !attr_set[dev]) {
    const cudaError_t e = cudaFuncSetAttribute(pre_attention_rows_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, 100 << 10);
    if (e != cudaSuccess) return fail(NVLLM_E_CUDA, "qk_norm_rope_store: set-up failed: %s", cudaGetErrorString(e));
    attr_set[dev] = true;
  }
  const int64_t grid = std::min<int64_t>(p.n_tokens, static_cast<int64_t>(sms) * blocks_per_sm);
  return launch_kernel("qk_norm_rope_store", pre_attention_rows_kernel<D>, dim3(static_cast<unsigned>(grid)), dim3(kRowWarps * 32),
                       static_cast<size_t>(kRowStages) * stage_bytes, stream, p, stage_bytes);
}

}  // namespace nvllm

extern "C" int nvllm_qk_norm_rope_store(void* qkv, int64_t row_stride, const int64_t* positions, const void* q_weight,
                                        const void* k_weight, const float* cos_sin_cache, int64_t max_position, float eps,
                                        const int32_t* slot_mapping, void* k_cache, void* v_cache, int64_t num_slots,
                                        int64_t n_tokens, int32_t num_q_heads, int32_t num_kv_heads, int32_t head_dim,
                                        void* stream) {
  using namespace nvllm;
  if (head_dim != 64 && head_dim != 128)
    return fail(NVLLM_E_GEOMETRY, "qk_norm_rope_store: head_dim=%d unsupported (64 or 128)", head_dim);
  if (num_q_heads <= 0 || num_kv_heads <= 0) return fail(NVLLM_E_GEOMETRY, "qk_norm_rope_store: head counts must be positive");
  if (n_tokens < 0 || max_position <= 0) return fail(NVLLM_E_GEOMETRY, "qk_norm_rope_store: n_tokens / max_position invalid");
  if (n_tokens == 0) return NVLLM_OK;
  if (!qkv || !positions || !cos_sin_cache) return fail(NVLLM_E_NULL, "qk_norm_rope_store: NULL pointer argument");
  if ((q_weight == nullptr) != (k_weight == nullptr))
    return fail(NVLLM_E_NULL, "qk_norm_rope_store: give both norm weights or neither");
  const int64_t width = static_cast<int64_t>(num_q_heads + 2 * num_kv_heads) * head_dim;
  if (row_stride < width) return fail(NVLLM_E_GEOMETRY, "qk_norm_rope_store: row stride smaller than (Hq+2Hkv)*D");
  if (row_stride % 8 || !aligned16(qkv)) return fail(NVLLM_E_ALIGN, "qk_norm_rope_store: qkv and its row stride must be 16-byte aligned");
  if (slot_mapping) {
    if (!k_cache || !v_cache || num_slots <= 0) return fail(NVLLM_E_NULL, "qk_norm_rope_store: slot_mapping given without caches");
    if (!aligned16(k_cache) || !aligned16(v_cache)) return fail(NVLLM_E_ALIGN, "qk_norm_rope_store: caches must be 16-byte aligned");
  }
  PreAttnParams p;
  p.status = status_word();
  if (!p.status) return fail(NVLLM_E_NO_DEVICE, "qk_norm_rope_store: no CUDA device is usable");
  p.qkv = static_cast<__nv_bfloat16*>(qkv);
  p.row_stride = row_stride;
  p.positions = positions;
  p.q_weight = static_cast<const __nv_bfloat16*>(q_weight);
  p.k_weight = static_cast<const __nv_bfloat16*>(k_weight);
  p.cos_sin = cos_sin_cache;
  p.max_position = max_position;
  p.eps = eps;
  p.slot_mapping = slot_mapping;
  p.k_cache = static_cast<__nv_bfloat16*>(k_cache);
  p.v_cache = static_cast<__nv_bfloat16*>(v_cache);
  p.num_slots = num_slots;
  p.n_tokens = n_tokens;
  p.hq = num_q_heads;
  p.hkv = num_kv_heads;
  p.tables_aligned = aligned16(cos_sin_cache) && aligned16(q_weight) && aligned16(k_weight);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  // Whole rows from 6 MB of them on, where the two forms cross in all three geometries (512 tokens of 12
  // KB, between 512 and 1024 of 8 KB, 2048 of 2.3 KB); below, a head per lane group, so that a decode
  // batch spreads over the chip and a lane's chain is as short as it can be (16 tokens: 1.7 us, 3.0 by
  // rows).  Blocks per SM: as many rings as its shared memory holds (1 KB of it goes with every block).
  const int sms = num_sms();
  const int64_t stage = (head_dim * 4 + width * 2 + 127) / 128 * 128;
  const int blocks_per_sm = static_cast<int>(std::min<int64_t>(16, (227 << 10) / (kRowStages * stage + 1024)));
  const bool rows = p.tables_aligned && sms > 0 && kRowStages * stage <= (100 << 10) && n_tokens * width * 2 >= kRowsFromBytes;
  if (rows)
    return head_dim == 128 ? launch_pre_attention_rows<128>(p, blocks_per_sm, static_cast<int>(stage), sms, st)
                           : launch_pre_attention_rows<64>(p, blocks_per_sm, static_cast<int>(stage), sms, st);
  return head_dim == 128 ? launch_pre_attention<128>(p, st) : launch_pre_attention<64>(p, st);
}
