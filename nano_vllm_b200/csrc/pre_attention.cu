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
// Bound by memory: 18 KB per token in the Qwen3-0.6B geometry.  A head is read and written in 16-byte
// pieces by D/8 neighbouring lanes (16 for head_dim 128), so a warp holds 256 / D heads and every
// access is a full 128-byte line; the rotation partner x[i +- D/2] sits D/16 lanes away and comes by
// shuffle, as packed bf16 (what is rotated has been rounded to bf16 already).  A lane group takes
// HPT heads of one token: their loads are all in flight before the first is used, and the token's
// cos / sin values (four times as many bytes as a head has) are fetched once for all of them.
// 16384 tokens (302 MB): 117 us with one warp per head and 4-byte accesses, 65 us so (105, 79 and 64 us
// with one, two and eight heads per group; below some 2400 tokens one head is the faster).
#include "common.cuh"

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

constexpr int kPreThreads = 256;

template <int D, int HPT>
__global__ void __launch_bounds__(kPreThreads) pre_attention_kernel(const PreAttnParams p) {
  pdl_prologue();  // lets the attention kernel that follows get its blocks resident early
  constexpr int LANES = D / 8;  // lanes of a head
  const int sub = threadIdx.x & (LANES - 1);
  const unsigned heads = p.hq + 2 * p.hkv, parts = (heads + HPT - 1) / HPT;
  const unsigned unit = blockIdx.x * (kPreThreads / LANES) + threadIdx.x / LANES;
  // The whole warp stays to the end (it shuffles); lane groups past the last unit do nothing else.
  const bool live = unit < p.n_tokens * parts;
  const unsigned tok = live ? unit / parts : 0, h0 = live ? (unit - tok * parts) * HPT : heads;
  __nv_bfloat16* row = p.qkv + tok * p.row_stride + sub * 8;

  uint4 raw[HPT];
#pragma unroll
  for (int j = 0; j < HPT; ++j)
    raw[j] = h0 + j < heads ? *reinterpret_cast<const uint4*>(row + static_cast<int64_t>(h0 + j) * D) : make_uint4(0, 0, 0, 0);

  int64_t pos = p.positions[tok];
  if (pos < 0 || pos >= p.max_position) pos = pos < 0 ? 0 : p.max_position - 1;
  int64_t slot = -1;
  if (p.slot_mapping && h0 + HPT > static_cast<unsigned>(p.hq) && live) {
    slot = p.slot_mapping[tok];
    if (slot >= p.num_slots) {
      if (sub == 0) atomicOr(p.status, NVLLM_STATUS_BAD_SLOT);
      slot = -1;
    }
  }
  const bool upper = sub >= LANES / 2;
  uint64_t c[4], s[4];
  load_table(p.cos_sin + pos * D + (sub % (LANES / 2)) * 8, p.tables_aligned, c);
  load_table(p.cos_sin + pos * D + D / 2 + (sub % (LANES / 2)) * 8, p.tables_aligned, s);
  if (!upper) {  // x1 cos - x2 sin in the lower half, x2 cos + x1 sin in the upper
#pragma unroll
    for (int i = 0; i < 4; ++i) s[i] ^= 0x8000000080000000ull;
  }

#pragma unroll
  for (int j = 0; j < HPT; ++j) {
    const int head = static_cast<int>(h0) + j;
    if (p.q_weight) {  // uniform over the launch
      uint64_t x[4];
      unpack8(raw[j], x);
      uint64_t sq = mul2(x[0], x[0]);
#pragma unroll
      for (int i = 1; i < 4; ++i) sq = fma2(x[i], x[i], sq);
      float ss, ss1;
      unpack2(sq, ss, ss1);
      ss += ss1;
#pragma unroll
      for (int sh = LANES / 2; sh > 0; sh >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, sh);
      if (head < p.hq + p.hkv) {
        const float rstd = rsqrtf(ss * (1.0f / D) + p.eps);
        const uint4 w = load_weights((head < p.hq ? p.q_weight : p.k_weight) + sub * 8, p.tables_aligned);
#pragma unroll
        for (int i = 0; i < 4; ++i) x[i] = mul2(x[i], pack2(rstd, rstd));
        const uint4 n = pack8(x);
        raw[j] = make_uint4(mul_bf16x2(n.x, w.x), mul_bf16x2(n.y, w.y), mul_bf16x2(n.z, w.z), mul_bf16x2(n.w, w.w));
      }
    }
    uint4 other;
    other.x = __shfl_xor_sync(0xffffffffu, raw[j].x, LANES / 2);
    other.y = __shfl_xor_sync(0xffffffffu, raw[j].y, LANES / 2);
    other.z = __shfl_xor_sync(0xffffffffu, raw[j].z, LANES / 2);
    other.w = __shfl_xor_sync(0xffffffffu, raw[j].w, LANES / 2);
    if (head < p.hq + p.hkv) {
      uint64_t x[4], y[4];
      unpack8(raw[j], x);
      unpack8(other, y);
#pragma unroll
      for (int i = 0; i < 4; ++i) x[i] = add2(mul2(x[i], c[i]), mul2(y[i], s[i]));
      raw[j] = pack8(x);
      *reinterpret_cast<uint4*>(row + static_cast<int64_t>(head) * D) = raw[j];
    }
    if (slot >= 0 && head >= p.hq && head < static_cast<int>(heads)) {
      __nv_bfloat16* cache = head < p.hq + p.hkv ? p.k_cache + (slot * p.hkv + (head - p.hq)) * D
                                                 : p.v_cache + (slot * p.hkv + (head - p.hq - p.hkv)) * D;
      *reinterpret_cast<uint4*>(cache + sub * 8) = raw[j];
    }
  }
}

template <int D, int HPT>
static int launch_pre_attention(const PreAttnParams& p, cudaStream_t stream) {
  const int64_t units = p.n_tokens * ((p.hq + 2 * p.hkv + HPT - 1) / HPT);
  constexpr int per_block = kPreThreads / (D / 8);
  if (units > 0x7fffffffLL) return fail(NVLLM_E_GEOMETRY, "qk_norm_rope_store: too many tokens for one launch");
  return launch_kernel("qk_norm_rope_store", pre_attention_kernel<D, HPT>,
                       dim3(static_cast<unsigned>((units + per_block - 1) / per_block)), dim3(kPreThreads), 0, stream, p);
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
  // Four heads per lane group once that still leaves every SM its 2048 threads; below, one head each,
  // so that a decode batch spreads over the chip and a lane's chain is as short as it can be.
  const int sms = num_sms();
  const int64_t lanes = n_tokens * (num_q_heads + 2 * num_kv_heads) * (head_dim / 8);
  const bool wide = lanes >= 4ll * 2048 * (sms > 0 ? sms : 1);
  if (head_dim == 128) return wide ? launch_pre_attention<128, 4>(p, st) : launch_pre_attention<128, 1>(p, st);
  return wide ? launch_pre_attention<64, 4>(p, st) : launch_pre_attention<64, 1>(p, st);
}
