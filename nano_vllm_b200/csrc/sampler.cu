// Token sampling in one pass over the logits.
//
// Stands where nano-vllm's Sampler.forward stands (nanovllm/layers/sampler.py:10-26), which
// spends eight elementwise / reduction launches over a [batch, vocab] fp32 copy of the logits:
//   greedy = argmax(logits);  probs = softmax(logits / T);
//   sample = argmax(probs / (Exponential(1) + 1e-10));  token = (T == 0) ? greedy : sample.
// argmax(p_i / e_i) is the Gumbel-max ("exponential race") way of drawing from p.  Since the
// softmax normaliser and the row maximum are common to a row, the same token is
//   argmax_i ( logit_i / T  -  ln(e_i + 1e-10) ),
// which needs neither the maximum nor the sum: one read of the row, no intermediate tensor.
//
// Two noise sources.  (1) `noise` given: e_i is read from the caller's [batch, vocab] fp32
// tensor; with the tensor the reference drew, the result is the reference's token (up to
// rounding when two candidates tie to ~1e-6 relative).  (2) `noise` NULL: e_i = -ln(1 - v)
// with v uniform in (0,1) from a Philox4x32-10 counter-based generator keyed by (seed) and
// counted by (row, position in the row, step); no state is kept between calls, the same
// (seed, step) reproduces the same tokens.
//
// A row is read by one thread-block cluster of 1 to 8 or 16 blocks of 256 to 768 threads, so that a decode batch of any
// size spreads evenly over the 148 SMs.  A thread takes groups of 16 bytes (8 bf16 or 4 fp32 logits), loaded one step ahead.  Each
// warp reduces to one candidate and puts it into the shared memory of the cluster's first block, where
// the largest is taken.  Ties go to the lowest index.
//
// What bounds it: not the one read of the logits (78 MB at batch 256, 12 us) but the instructions
// per element: the generator alone, at 768 threads to an SM and without a load, takes 24.7 us of the 43.5 there, 21 of
// them its 18 wide products for four logits (29 a clock and SM).  Ten Philox rounds for four elements and two logarithms for each came to 74 us there
// (now 43.5; greedy rows 32 -> 16; batch 1, 12.7 -> 5.7).  The logarithms are only needed for elements that
// can still win: since e >= v, where v is the uniform
// draw, element i can beat a score b only if v < exp(x_i - b), x_i = logit_i / T.  One exponential of
// the group's largest x and the smallest of its draws decide that for the whole group, against the
// best score that any warp of the block has seen; only groups that pass (a few per warp and row)
// compute their scores.  A warp whose groups cannot pass even with the smallest possible draw
// (x < b - 22) skips the generator as well, which is where most of the vocabulary of a peaked
// distribution ends.  Greedy rows compare the group's maximum with the thread's best, two packed bf16 at a time.
//
// Groups start at multiples of four global positions (the generator's counter).  Where such a
// group does not start on a 16-byte boundary (rows of an odd vocabulary, slices), it is put together
// from words (greedy fp32 rows: starts on one); the up to fifteen elements around the whole groups go one at a time.
//
// Tensor parallelism: nano-vllm's LM head leaves every rank with the logits of its own slice of
// the vocabulary and then gathers all slices on rank 0 and concatenates them
// (nanovllm/layers/embed_head.py:78-87) before it samples.  The candidate form of this kernel
// makes that traffic unnecessary: every rank reduces its slice to one (score, global index)
// candidate per row, packed into an int64 whose signed order is "higher score first, then lower
// index"; a MAX over the ranks (8 bytes per row) then picks the token that the one-rank kernel
// would have picked from the concatenated row, because the noise is generated from the global
// index.  nvllm_sample_unpack turns the winning candidates into token ids.
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>
#include <mutex>
#include <type_traits>
#include <utility>

#include "common.cuh"

namespace nvllm {

struct SampleParams {
  const void* logits;
  int64_t row_stride;
  const float* temperatures;
  const float* noise;  // nullable
  int64_t noise_stride;
  uint64_t step;
  uint2 key[10];            // the generator's keys of its ten rounds, from the seed
  int64_t* tokens;          // token ids, or packed candidates when `candidates` is set
  int vocab;                // elements in a row of `logits`
  int64_t offset;           // global vocabulary index of element 0 of a row
  int candidates;
};

// Float bits as a signed integer of the same order.
__device__ __forceinline__ int ordered(float x) {
  const int i = __float_as_int(x);
  return i >= 0 ? i : i ^ 0x7fffffff;
}
__device__ __forceinline__ float from_ordered(int i) { return __int_as_float(i >= 0 ? i : i ^ 0x7fffffff); }

// (score, index) as one int64 that orders like "higher score, then lower index".
__device__ __forceinline__ long long pack_candidate(float score, int idx) {
  const int s = ordered(score);
  return (static_cast<long long>(s) << 32) | static_cast<long long>(0xffffffffu - static_cast<unsigned int>(idx));
}

__device__ __forceinline__ int64_t candidate_index(long long packed) {
  const unsigned int idx = 0xffffffffu - static_cast<unsigned int>(packed & 0xffffffffll);
  return idx == 0x7fffffffu ? 0 : static_cast<int64_t>(idx);
}

// Philox4x32 with 10 rounds (Salmon et al., "Parallel random numbers: as easy as 1, 2, 3", SC'11),
// for counters (c0, row, step lo, step hi) of which only c0 differs between the calls of a thread:
// one product of round 1 and one of round 2 do not depend on it and are made once.  High and low
// words are separate multiplications on purpose: the 64-bit product is one instruction but slower
// (64 us against 56 for the whole kernel at batch 256).
// The round keys come with the kernel's parameters, where an instruction can read them in place.
struct Philox {
  static constexpr uint32_t M0 = 0xD2511F53u, M1 = 0xCD9E8D57u;
  const uint2 (&key)[10];
  uint32_t a, b, c, d;  // key and counter words that are the same for every c0
  __device__ __forceinline__ Philox(const uint2 (&keys)[10], uint32_t row, uint64_t step) : key(keys) {
    const uint32_t lo = static_cast<uint32_t>(step), hi = static_cast<uint32_t>(step >> 32);
    a = hi ^ key[0].y;                            // round 1: z = hi(M0 c0) ^ a, w = lo(M0 c0)
    const uint32_t x1 = __umulhi(M1, lo) ^ row ^ key[0].x;
    b = (M1 * lo) ^ key[1].x;              // round 2: x = hi(M1 z) ^ b, y = lo(M1 z)
    c = __umulhi(M0, x1) ^ key[1].y;       //          z = w ^ c
    d = M0 * x1;                               //          w = d
  }
  __device__ __forceinline__ uint4 operator()(uint32_t c0) const {
    const uint32_t z1 = __umulhi(M0, c0) ^ a, w1 = M0 * c0;
    uint4 s = make_uint4(__umulhi(M1, z1) ^ b, M1 * z1, w1 ^ c, d);
#pragma unroll
    for (int r = 2; r < 10; ++r) {
      const uint32_t hi0 = __umulhi(M0, s.x), lo0 = M0 * s.x;
      const uint32_t hi1 = __umulhi(M1, s.z), lo1 = M1 * s.z;
      s = make_uint4(hi1 ^ s.y ^ key[r].x, lo1, hi0 ^ s.w ^ key[r].y, lo0);
    }
    return s;
  }
};

// ln of an Exponential(1) draw made from 32 random bits.  v = (bits + 0.5) / 2^32 is uniform in
// (0,1) and e = -ln(1 - v); for small v the series keeps the relative precision that 1 - v
// would lose (small e decides which unlikely token wins, large e never matters).
__device__ __forceinline__ float ln_exponential(uint32_t bits) {
  const float v = (static_cast<float>(bits >> 8) + 0.5f) * 5.9604644775390625e-08f;  // 24 bits, never 0 or 1
  float e;
  if (v < 0.03125f) {
    // the low 8 bits refine v where it is small enough for them to matter
    const float vf = (static_cast<float>(bits) + 0.5f) * 2.3283064365386963e-10f;
    e = vf * (1.f + vf * (0.5f + vf * (0.33333334f + vf * 0.25f)));
  } else {
    e = -__logf(1.f - v);
  }
  return __logf(e);
}

struct Best {
  float score;
  int idx;
};
__device__ __forceinline__ void take(Best& b, float s, int i) {
  // NaN never wins; ties keep the lower index
  if (s > b.score || (s == b.score && i < b.idx)) {
    b.score = s;
    b.idx = i;
  }
}
// Same for the groups of a thread, which it visits in rising index order.
__device__ __forceinline__ void take_next(Best& b, float s, int i) {
  if (s > b.score) {
    b.score = s;
    b.idx = i;
  }
}

// A group is one 16-byte piece of a row: its elements as fp32, and their maximum (NaN ignored).
template <typename T>
struct Group;
template <>
struct Group<__nv_bfloat16> {
  static constexpr int N = 8;
  static __device__ __forceinline__ void unpack(const uint4& w, float (&x)[N]) {
    const uint32_t u[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      x[2 * i] = __uint_as_float(u[i] << 16);
      x[2 * i + 1] = __uint_as_float(u[i] & 0xffff0000u);
    }
  }
  static __device__ __forceinline__ float max(const uint4& w) {
    auto h = [](uint32_t u) { return *reinterpret_cast<__nv_bfloat162*>(&u); };
    const __nv_bfloat162 m = __hmax2(__hmax2(h(w.x), h(w.y)), __hmax2(h(w.z), h(w.w)));
    return fmaxf(__low2float(m), __high2float(m));
  }
};
template <>
struct Group<float> {
  static constexpr int N = 4;
  static __device__ __forceinline__ void unpack(const uint4& w, float (&x)[N]) {
    x[0] = __uint_as_float(w.x);
    x[1] = __uint_as_float(w.y);
    x[2] = __uint_as_float(w.z);
    x[3] = __uint_as_float(w.w);
  }
  static __device__ __forceinline__ float max(const uint4& w) {
    return fmaxf(fmaxf(__uint_as_float(w.x), __uint_as_float(w.y)), fmaxf(__uint_as_float(w.z), __uint_as_float(w.w)));
  }
};

// Calls f(pieces, first group, stride between the pieces' groups, full) for this thread's share of the
// `n_groups` groups of a row that start at `first`, C pieces at a time; the next C are loaded before
// the current ones are looked at.  All lanes of a warp make the same calls.  full is a constant: true
// where every piece of every lane of the warp is a group, else pieces past the end are zero.
// Pieces of a row that does not start on a 16-byte boundary come as the words that hold them, and are shifted by half a word,
// where that is needed, when their turn comes: shifted as they were loaded they held every step up for
// its own load (256 rows of 151643 bf16 54.7 -> 48.5 us, 512 102 -> 85, 300 of 50257 28.4 -> 26.1).
struct Words {
  uint32_t u[5];
};

template <bool ALIGNED, int C, typename T, class F>
__device__ __forceinline__ void for_groups(const T* first, int n_groups, int tid, int nthreads, F&& f) {
  using Piece = std::conditional_t<ALIGNED, uint4, Words>;
  const int lane = tid & 31;
  const uint4* base = reinterpret_cast<const uint4*>(first);
  const uint32_t* words = reinterpret_cast<const uint32_t*>(reinterpret_cast<uintptr_t>(first) & ~uintptr_t{3});
  const bool across = sizeof(T) == 2 && (reinterpret_cast<uintptr_t>(first) & 2);  // elements lie across two words
  auto load = [&](Piece (&piece)[C], int g, auto full) {
#pragma unroll
    for (int c = 0; c < C; ++c, g += nthreads) {
      const bool live = decltype(full)::value || g < n_groups;
      if constexpr (ALIGNED) {
        piece[c] = live ? __ldg(base + g) : make_uint4(0, 0, 0, 0);
      } else {
#pragma unroll
        for (int i = 0; i < 5; ++i) piece[c].u[i] = live && (i < 4 || across) ? __ldg(words + 4 * static_cast<int64_t>(g) + i) : 0;
      }
    }
  };
  auto whole = [&](const Piece& p) {
    if constexpr (ALIGNED) {
      return p;
    } else {
      uint32_t u[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) u[i] = across ? __funnelshift_r(p.u[i], p.u[i + 1], 16) : p.u[i];
      return make_uint4(u[0], u[1], u[2], u[3]);
    }
  };
  const int step = C * nthreads;
  uint4 raw[C];
  Piece next[C];
  int g = tid;
  const int n_full = n_groups - (C - 1) * nthreads - (31 - lane);  // g below this: a full call (the same for all lanes)
  if (g < n_full) load(next, g, std::true_type{});
  while (g < n_full) {
#pragma unroll
    for (int c = 0; c < C; ++c) raw[c] = whole(next[c]);
    if (g + step < n_full) load(next, g + step, std::true_type{});
    f(raw, g, nthreads, std::true_type{});
    g += step;
  }
  for (; g - lane < n_groups; g += step) {
    load(next, g, std::false_type{});
#pragma unroll
    for (int c = 0; c < C; ++c) raw[c] = whole(next[c]);
    f(raw, g, nthreads, std::false_type{});
  }
}

constexpr int kMaxCluster = 16;

template <typename T>
__global__ void __launch_bounds__(1024, 1) sample_kernel(const SampleParams p) {
  using G = Group<T>;
  constexpr int N = G::N;
  namespace cg = cooperative_groups;
  pdl_wait();
  cg::cluster_group cluster = cg::this_cluster();
  auto started = cluster.barrier_arrive();  // waited for before another block's shared memory is written
  const int csize = static_cast<int>(cluster.num_blocks()), crank = static_cast<int>(cluster.block_rank());
  const int row = blockIdx.x / csize;
  const int tid = crank * blockDim.x + threadIdx.x;  // thread index within the row's cluster
  const int nthreads = csize * blockDim.x;
  const T* x = static_cast<const T*>(p.logits) + static_cast<int64_t>(row) * p.row_stride;
  const float* nz = p.noise ? p.noise + static_cast<int64_t>(row) * p.noise_stride : nullptr;
  const float t = p.temperatures[row];
  const bool greedy = !(t > 0.f) && !(t < 0.f);  // T == 0 (or NaN): plain argmax, as torch.where(T == 0, ...)
  const float inv_t = greedy ? 1.f : 1.f / t;
  const Philox draw4(p.key, static_cast<uint32_t>(row), p.step);  // unique per element and call
  __shared__ int s_best;  // best score of the block so far, ordered()
  __shared__ long long s_candidates[kMaxCluster * 32];  // block 0 of the cluster: one per warp of the row
  if (threadIdx.x == 0) s_best = ordered(-INFINITY);
  __syncthreads();

  Best best{-INFINITY, 0x7fffffff};
  const int off = static_cast<int>(p.offset);
  // Whole groups of this row: they start at multiples of four global positions, the generator's counter.  Where nothing is
  // generated, fp32 ones start on 16-byte boundaries instead: put together from four words each they held the loads up
  // (512 greedy rows of 151643 fp32 59.7 -> 49.1 us, 256 of 50257 11.7 -> 7.7).
  int lead = (4 - (off & 3)) & 3;
  if (sizeof(T) == 4 && greedy) lead = static_cast<int>((16u - (reinterpret_cast<uintptr_t>(x) & 15u)) & 15u) / static_cast<int>(sizeof(T));
  const int n_groups = p.vocab > lead ? (p.vocab - lead) / N : 0;
  const T* first = x + lead;

  auto scan = [&](auto aligned) {
    constexpr bool A = decltype(aligned)::value;
    if (greedy) {
      for_groups<A, 4>(first, n_groups, tid, nthreads, [&](const uint4 (&raw)[4], int g, int stride, auto full) {
#pragma unroll
        for (int c = 0; c < 4; ++c, g += stride) {
          if ((!decltype(full)::value && g >= n_groups) || !(G::max(raw[c]) > best.score)) continue;
          float e[N];
          G::unpack(raw[c], e);
#pragma unroll
          for (int k = 0; k < N; ++k) take_next(best, e[k], off + lead + g * N + k);
        }
      });
    } else if (nz) {
      for_groups<A, 1>(first, n_groups, tid, nthreads, [&](const uint4 (&raw)[1], int g, int, auto full) {
        if (!decltype(full)::value && g >= n_groups) return;
        float e[N];
        G::unpack(raw[0], e);
        const float* z = nz + lead + g * N;
#pragma unroll
        for (int k = 0; k < N; ++k) take_next(best, e[k] * inv_t - __logf(z[k] + 1e-10f), off + lead + g * N + k);
      });
    } else {
      // log2 of 2^32 times the largest v with which x reaches a score b: x log2(e) / T - bar_of(b).  The slack
      // covers the rounding of the scores, of the exponential and of v.
      const float x_scale = inv_t * 1.4426950408889634f;
      auto bar_of = [&](float b) { return t < 0.f ? -INFINITY : fmaf(b, 1.4426950408889634f, -32.01f - 1e-6f * fabsf(b)); };
      // draws up to this can win; NaN (nothing seen yet, infinities) and T < 0 let everything pass
      auto limit_of = [&](const uint4& raw, float bar) { return fast_exp2(fmaf(G::max(raw), x_scale, -bar)); };
      float bar = bar_of(-INFINITY);
      int seen = ordered(-INFINITY);
      // One group at a time: two, with twice as many generator chains in flight, were slower below some 400
      // rows, and so were fewer registers and more warps.
      for_groups<A, 1>(first, n_groups, tid, nthreads, [&](const uint4 (&raw)[1], int g, int, auto full) {
        const bool live = decltype(full)::value || g < n_groups;
        const int now = *static_cast<volatile int*>(&s_best);
        if (now != seen) {
          seen = now;
          bar = bar_of(from_ordered(now));
        }
        float limit = limit_of(raw[0], bar);
        if (!__any_sync(0xffffffffu, live && !(limit < 0.25f))) return;
        const int pos = off + lead + g * N;
        uint32_t bits[N];
#pragma unroll
        for (int h = 0; h < N / 4; ++h) {
          const uint4 r = draw4(static_cast<uint32_t>(pos >> 2) + h);
          bits[4 * h] = r.x; bits[4 * h + 1] = r.y; bits[4 * h + 2] = r.z; bits[4 * h + 3] = r.w;
        }
        float e[N];
        if (seen == ordered(-INFINITY)) {
          // Nothing is known of the row yet: take a bar from these elements.  -ln(e) >= -ln(v) - 0.33 for
          // v < 1/2 (e <= 1.39 v), and the exponent and mantissa bits of v read as a number give log2(v)
          // to within 0.09, so this is a score that some element reaches, found without logarithms.
          float reach = -INFINITY;
          if (live) {
            G::unpack(raw[0], e);
#pragma unroll
            for (int k = 0; k < N; ++k) {
              const float log2v = fmaf(static_cast<float>(__float_as_int(static_cast<float>(bits[k]) + 0.5f)),
                                       1.1920928955078125e-07f, -159.f);
              const float s = fmaf(log2v + 0.1f, -0.69314718f, fmaf(e[k], inv_t, -0.33f));
              if (bits[k] < 0x80000000u) reach = fmaxf(reach, s);
            }
          }
          const int reached = __reduce_max_sync(0xffffffffu, ordered(reach));
          if ((threadIdx.x & 31) == 0) atomicMax(&s_best, reached);
          limit = limit_of(raw[0], bar_of(from_ordered(reached)));
        }
        const uint32_t below = limit < 4.2e9f ? __float2uint_ru(limit) : 0xffffffffu;  // NaN: everything passes
        uint32_t least = min(min(bits[0], bits[1]), min(bits[2], bits[3]));
        if constexpr (N == 8) least = min(least, min(min(bits[4], bits[5]), min(bits[6], bits[7])));
        const bool pass = live && least <= below;
        if (!__any_sync(0xffffffffu, pass)) return;
        if (pass) {
          G::unpack(raw[0], e);
#pragma unroll
          for (int k = 0; k < N; ++k)
            if (bits[k] <= below) take_next(best, e[k] * inv_t - ln_exponential(bits[k]), pos + k);
        }
        const int warp_best = __reduce_max_sync(0xffffffffu, ordered(best.score));
        if ((threadIdx.x & 31) == 0 && warp_best > now) atomicMax(&s_best, warp_best);
      });
    }
  };
  if ((reinterpret_cast<uintptr_t>(first) & 15u) == 0) scan(std::true_type{});
  else scan(std::false_type{});
  // the elements before and after the whole groups, one at a time, same counters
  const int n_edge = p.vocab - n_groups * N, head = min(lead, p.vocab);
  for (int k = tid; k < n_edge; k += nthreads) {
    const int i = k < head ? k : k + n_groups * N;
    float s = static_cast<float>(x[i]) * inv_t;
    if (!greedy) {
      if (nz) {
        s -= __logf(nz[i] + 1e-10f);
      } else {
        const int gi = off + i;  // global position
        const uint4 r = draw4(static_cast<uint32_t>(gi >> 2));
        const uint32_t w[4] = {r.x, r.y, r.z, r.w};
        s -= ln_exponential(w[gi & 3]);
      }
    }
    take(best, s, off + i);
  }

  // Argmax of the row: by shuffle inside a warp, then every warp of the cluster puts its candidate into
  // block 0's shared memory, and one warp there takes the largest.
#pragma unroll
  for (int sh = 16; sh > 0; sh >>= 1) {
    const float s = __shfl_xor_sync(0xffffffffu, best.score, sh);
    const int i = __shfl_xor_sync(0xffffffffu, best.idx, sh);
    take(best, s, i);
  }
  // The next kernel's blocks start when the last block here gets to its merge: started any earlier they land on the SMs that
  // happen to be free first, two on one and none on the next (32 rows 17.8 us instead of 12.9).
  pdl_trigger();
  cluster.barrier_wait(std::move(started));
  const int lt = threadIdx.x, warps = static_cast<int>(blockDim.x) >> 5;
  if ((lt & 31) == 0)
    cluster.map_shared_rank(s_candidates, 0)[crank * warps + (lt >> 5)] = pack_candidate(best.score == 0.f ? 0.f : best.score, best.idx);
  cluster.sync();
  if (crank != 0 || lt >= 32) return;
  long long top = s_candidates[0];
  for (int k = lt; k < csize * warps; k += 32) top = max(top, s_candidates[k]);
#pragma unroll
  for (int sh = 16; sh > 0; sh >>= 1) top = max(top, __shfl_xor_sync(0xffffffffu, top, sh));
  // a row of NaN / -inf only: token 0, like an argmax over equal values (after the merge, for
  // candidates: the sentinel index loses against any real candidate of another rank)
  if (lt == 0) p.tokens[row] = p.candidates ? top : candidate_index(top);
}

__global__ void sample_unpack_kernel(const long long* packed, int64_t* tokens, int batch) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= batch) return;
  tokens[b] = candidate_index(packed[b]);
}

constexpr int kThreads = 256, kPortableCluster = 8;

struct Shape {
  int blocks, threads;  // to a row, to a block
};

// Blocks of 256 threads to a row in powers of two: as few as give every SM three, in waves where that is more than it holds.
// No more than the row has work for.
static Shape in_waves(int batch, int vocab, int sms) {
  int csize = 1;
  while (csize < kPortableCluster && static_cast<int64_t>(batch) * csize < 3ll * sms && vocab >= 2 * csize * kThreads * 8) csize *= 2;
  return {csize, kThreads};
}

// How a launch is laid out.  The generator keeps an SM busy from some 24 warps on, so a launch takes as long as the SM with
// most rows to read, in whole or in part, and what counts is to spread them evenly and at once.  Blocks of 768 threads
// stand one to an SM, so that as many clusters as the device can hold of them are spread evenly by force; 384 stand two to
// an SM, 256 four.  Clusters are counted as the device counts them: one lies within a group of SMs, and what is left of a
// group is no use to it (of six blocks to an SM each, 148 SMs hold 22).  Blocks of 512 threads are spread evenly only where a
// cluster has one or two, 256 where it has two and every thread something to read.  The cost of a form is what the fullest
// SM's share of sampled bf16 rows of 151936 logits took in it, over that of 512 threads; fp32 and greedy rows go by the same,
// as the host does not know the temperatures.  Where it leads to no form that is even, powers of two in waves (in_waves):
// more than two rows to an SM (300 rows 57 us, 65 at once, 400 65 and 76; waves of blocks of 512 threads sample 512 in 76
// instead of 85, but take 29.3 instead of 25.7 for 450 greedy ones), and long ones of which SMs would have one or two (200
// 36.4, 41.7 at once; fp32 45.6, 50.5, though greedy 25.1, 22.4).  Rows shorter than kLongRow have too little for the merges of
// four blocks of 256 threads and more (112 rows of 32000 10.2 -> 8.7 us, of 18992 greedy fp32 4.8 -> 4.0).
// Blocks that are not spread by force land 15 % unevenly: with 1 for the 1.15 below 200 sampled rows take 40.8 us instead of 38.3
// (greedy 14.5 instead of 17.1), over 480 launches 1, 1.15 and 1.3 are the same to 0.1 %.
// All for 151936 logits and T = 0.6 unless said, in waves -> now, us: 1 row 6.05 -> 5.4, 16 10.35 -> 8.15, 64 16.1 -> 14.4, 100 24.8 ->
// 21.7, 148 30.6 -> 23.6, 180 35.6 -> 31.4, 256 43.9 -> 42.3.  Of 980 launches (1-512 rows of 1000-151936 logits of both types,
// sampled and greedy) in a chain the mean is 11 % faster; 32 are 4 % slower or more, four of them by over 0.4 us (56 greedy
// fp32 rows of 18992 and 32000, 150 and 180 sampled ones of 4096) and 222 greedy bf16 rows of 151936 (11.2 -> 12.5).
struct Form {
  int threads, per_sm, least, most;  // of a block; blocks of it on an SM; blocks to a row
  double cost;                       // of a row, relative to 512 threads
};
constexpr Form kForms[] = {{768, 1, 1, 8, 1.05}, {512, 2, 1, 1, 1.0}, {512, 2, 2, 2, 1.07}, {384, 2, 3, 8, 1.07}, {256, 4, 3, 8, 1.17}, {256, 4, 1, 2, 1.05}};
static_assert(sizeof(kForms) / sizeof(kForms[0]) == NVLLM_SAMPLE_FORMS, "as the header says");
constexpr int kSixteen = 0;              // clusters of sixteen are counted in this form, one block to an SM, and launched with
constexpr int kSixteenThreads = 512;     // fewer threads: 5.65 us for one row, 5.9 with 768
constexpr int kFull = 768;               // threads that keep an SM busy
constexpr int64_t kLongRow = 8192;       // groups

// Clusters of every size that a device holds at a time, in every form; 0: it does not say.
struct Rooms {
  int of[NVLLM_SAMPLE_FORMS][kMaxCluster + 1];
};

static Shape shape_of(int batch, int vocab, int64_t vocab_offset, bool fp32, int sms, const Rooms& rooms) {
  const Shape waves = in_waves(batch, vocab, sms);
  if (rooms.of[kSixteen][2] <= 0 || batch > 2 * sms) return waves;
  const int64_t lead = (4 - (vocab_offset & 3)) & 3, groups = std::max<int64_t>(0, (vocab - lead) / (fp32 ? 4 : 8));
  Shape best{0, 0};
  double least = 0;  // of the groups that the fullest SM has to read
  auto offer = [&](const Form& form, int c, int threads, double per_sm) {  // per_sm: blocks on the fullest SM
    if (form.per_sm == 1)  // no more threads than a short row has groups
      threads = static_cast<int>(std::min<int64_t>(threads, std::max<int64_t>(kThreads, (groups + 32 * c - 1) / (32 * c) * 32)));
    double work = std::max<double>(static_cast<double>(groups), c * threads) * form.cost * per_sm / c;
    if (form.per_sm > 1) work *= std::max(1.0, kFull / (per_sm * threads));
    if (!best.blocks || work < least) best = {c, threads}, least = work;
  };
  if (rooms.of[kSixteen][kMaxCluster] >= batch) offer(kForms[kSixteen], kMaxCluster, kSixteenThreads, 1);
  for (int f = 0; f < NVLLM_SAMPLE_FORMS; ++f) {
    const Form& form = kForms[f];
    for (int c = form.least; c <= form.most; ++c) {
      if (form.threads == kThreads && c > 3 && groups < kLongRow) continue;
      const int64_t room = c == 1 ? static_cast<int64_t>(sms) * form.per_sm : rooms.of[f][c];
      const bool spread = c == 1 || (c * form.threads == 512 && groups >= 512);  // more evenly than an SM may hold of them
      if (room >= batch) offer(form, c, form.threads, spread ? std::min<double>(form.per_sm, std::ceil(1.15 * batch * c / sms)) : form.per_sm);
    }
  }
  // Between one and two long rows to an SM, where every such form leaves SMs with two rows beside SMs with one: in waves
  if (groups >= kLongRow && batch > sms) {
    const double filled = static_cast<double>(batch) * waves.blocks / (4.0 * sms);  // of what the SMs hold at a time
    const double rows = waves.blocks == 4 ? 1.575 + 0.882 * (filled - 1) : waves.blocks == 2 ? 2.19 - 0.8 * (1 - filled) : 4;
    if (rows * static_cast<double>(groups) < least) return waves;
  }
  return best;
}

template <typename T>
static const Rooms& rooms_of_device() {
  static Rooms known[64];
  static std::once_flag asked[64];
  static const Rooms none{};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
    (void)cudaGetLastError();
    return none;
  }
  std::call_once(asked[dev], [&] {
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    auto ask = [&](int f, int c) {
      int clusters = 0;
      attr[0].val.clusterDim.x = c;
      cfg.gridDim = dim3(c, 1, 1);
      cfg.blockDim = dim3(kForms[f].threads, 1, 1);
      if (cudaOccupancyMaxActiveClusters(&clusters, sample_kernel<T>, &cfg) != cudaSuccess) (void)cudaGetLastError();
      else known[dev].of[f][c] = clusters;
    };
    for (int f = 0; f < NVLLM_SAMPLE_FORMS; ++f)
      for (int c = std::max(2, kForms[f].least); c <= kForms[f].most; ++c) ask(f, c);
    // more than the portable eight blocks have to be allowed
    if (cudaFuncSetAttribute(sample_kernel<T>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess) ask(kSixteen, kMaxCluster);
    else (void)cudaGetLastError();
  });
  return known[dev];
}

static int sample_launch(const void* logits, int32_t logits_are_fp32, int64_t row_stride, const float* temperatures,
                         const float* exponential_noise, int64_t noise_row_stride, uint64_t seed, uint64_t step,
                         int64_t vocab_offset, int candidates, int64_t* tokens, int32_t batch, int32_t vocab, void* stream);

}  // namespace nvllm

extern "C" int nvllm_sample_plan(int32_t batch, int32_t vocab, int32_t num_sms, int32_t largest_cluster) {
  using namespace nvllm;
  if (batch < 0 || vocab <= 0 || num_sms <= 0) return fail(NVLLM_E_GEOMETRY, "sample_plan: batch=%d vocab=%d num_sms=%d invalid", batch, vocab, num_sms);
  const int c = in_waves(batch, vocab, num_sms).blocks;
  const bool sixteen = c == kPortableCluster && largest_cluster >= kMaxCluster && vocab >= kMaxCluster * kThreads * 8 &&
                       static_cast<int64_t>(batch) * kMaxCluster <= num_sms;
  return sixteen ? kMaxCluster : c;
}

extern "C" int nvllm_sample_layout(int32_t batch, int32_t vocab, int64_t vocab_offset, int32_t logits_are_fp32, int32_t num_sms,
                                   const int32_t* clusters, int32_t* blocks, int32_t* threads) {
  using namespace nvllm;
  if (batch < 0 || vocab <= 0 || vocab_offset < 0 || num_sms < 0 || (!num_sms && clusters))
    return fail(NVLLM_E_GEOMETRY, "sample_layout: batch=%d vocab=%d num_sms=%d invalid", batch, vocab, num_sms);
  if (!blocks || !threads) return fail(NVLLM_E_NULL, "sample_layout: NULL pointer argument");
  Rooms rooms{};
  if (clusters) std::copy(clusters, clusters + NVLLM_SAMPLE_FORMS * (kMaxCluster + 1), &rooms.of[0][0]);
  else if (!num_sms) rooms = logits_are_fp32 ? rooms_of_device<float>() : rooms_of_device<__nv_bfloat16>();
  const int sms = num_sms ? num_sms : nvllm::num_sms();
  if (sms <= 0) return fail(NVLLM_E_NO_DEVICE, "sample_layout: no CUDA device is usable");
  const Shape shape = shape_of(batch, vocab, vocab_offset, logits_are_fp32, sms, rooms);
  *blocks = shape.blocks;
  *threads = shape.threads;
  return NVLLM_OK;
}

extern "C" int nvllm_sample_tokens(const void* logits, int32_t logits_are_fp32, int64_t row_stride,
                                   const float* temperatures, const float* exponential_noise, int64_t noise_row_stride,
                                   uint64_t seed, uint64_t step, int64_t* tokens, int32_t batch, int32_t vocab,
                                   void* stream) {
  return nvllm::sample_launch(logits, logits_are_fp32, row_stride, temperatures, exponential_noise, noise_row_stride, seed, step,
                              0, 0, tokens, batch, vocab, stream);
}

extern "C" int nvllm_sample_candidates(const void* logits, int32_t logits_are_fp32, int64_t row_stride,
                                       const float* temperatures, const float* exponential_noise, int64_t noise_row_stride,
                                       uint64_t seed, uint64_t step, int64_t vocab_offset, int64_t* candidates, int32_t batch,
                                       int32_t vocab, void* stream) {
  using namespace nvllm;
  if (vocab_offset < 0 || vocab_offset + vocab > 0x7ffffffell)
    return fail(NVLLM_E_GEOMETRY, "sample_candidates: vocab_offset=%lld invalid", (long long)vocab_offset);
  return sample_launch(logits, logits_are_fp32, row_stride, temperatures, exponential_noise, noise_row_stride, seed, step,
                       vocab_offset, 1, candidates, batch, vocab, stream);
}

extern "C" int nvllm_sample_unpack(const int64_t* candidates, int64_t* tokens, int32_t batch, void* stream) {
  using namespace nvllm;
  if (batch < 0) return fail(NVLLM_E_GEOMETRY, "sample_unpack: batch=%d invalid", batch);
  if (batch == 0) return NVLLM_OK;
  if (!candidates || !tokens) return fail(NVLLM_E_NULL, "sample_unpack: NULL pointer argument");
  if (reinterpret_cast<uintptr_t>(candidates) % 8 || reinterpret_cast<uintptr_t>(tokens) % 8)
    return fail(NVLLM_E_ALIGN, "sample_unpack: pointers must be 8-byte aligned");
  sample_unpack_kernel<<<(batch + 255) / 256, 256, 0, static_cast<cudaStream_t>(stream)>>>(
      reinterpret_cast<const long long*>(candidates), tokens, batch);
  count_launch();
  return check_launch("sample_unpack launch");
}

namespace nvllm {
static int sample_launch(const void* logits, int32_t logits_are_fp32, int64_t row_stride, const float* temperatures,
                         const float* exponential_noise, int64_t noise_row_stride, uint64_t seed, uint64_t step,
                         int64_t vocab_offset, int candidates, int64_t* tokens, int32_t batch, int32_t vocab, void* stream) {
  if (batch < 0 || vocab <= 0) return fail(NVLLM_E_GEOMETRY, "sample_tokens: batch=%d vocab=%d invalid", batch, vocab);
  if (batch == 0) return NVLLM_OK;
  if (!logits || !temperatures || !tokens) return fail(NVLLM_E_NULL, "sample_tokens: NULL pointer argument");
  if (row_stride < vocab || (exponential_noise && noise_row_stride < vocab))
    return fail(NVLLM_E_GEOMETRY, "sample_tokens: a row stride is smaller than vocab");
  const size_t esz = logits_are_fp32 ? 4 : 2;
  if (reinterpret_cast<uintptr_t>(logits) % esz || reinterpret_cast<uintptr_t>(tokens) % 8 ||
      reinterpret_cast<uintptr_t>(temperatures) % 4 || reinterpret_cast<uintptr_t>(exponential_noise) % 4)
    return fail(NVLLM_E_ALIGN, "sample_tokens: a pointer is not aligned to its element size");
  SampleParams p;
  p.logits = logits;
  p.row_stride = row_stride;
  p.temperatures = temperatures;
  p.noise = exponential_noise;
  p.noise_stride = noise_row_stride;
  for (int r = 0; r < 10; ++r)
    p.key[r] = make_uint2(static_cast<uint32_t>(seed) + r * 0x9E3779B9u, static_cast<uint32_t>(seed >> 32) + r * 0xBB67AE85u);
  p.step = step;
  p.tokens = tokens;
  p.vocab = vocab;
  p.offset = vocab_offset;
  p.candidates = candidates;
  const int sms = num_sms();
  if (sms <= 0) return fail(NVLLM_E_NO_DEVICE, "sample_tokens: no CUDA device is usable");
  const Rooms& rooms = logits_are_fp32 ? rooms_of_device<float>() : rooms_of_device<__nv_bfloat16>();
  const Shape shape = shape_of(batch, vocab, vocab_offset, logits_are_fp32, sms, rooms);
  const int csize = shape.blocks;
  const int64_t blocks = static_cast<int64_t>(batch) * csize;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(blocks), 1, 1);
  cfg.blockDim = dim3(shape.threads, 1, 1);
  cfg.dynamicSmemBytes = 0;
  cfg.stream = static_cast<cudaStream_t>(stream);
  auto kernel = logits_are_fp32 ? sample_kernel<float> : sample_kernel<__nv_bfloat16>;
  cudaLaunchAttribute attr[2];
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = csize;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, p);
  if (e != cudaSuccess) {
    (void)cudaGetLastError();
    return fail(NVLLM_E_CUDA, "sample_tokens launch: %s", cudaGetErrorString(e));
  }
  count_launch();
  return check_launch("sample_tokens launch");
}
}  // namespace nvllm
