// Tile geometry, barrier roles and the bounded wait shared by the tcgen05 prefill kernels.
#pragma once

#include "common.cuh"
#include "sm100.cuh"

namespace nvllm {

namespace tc {
constexpr int BM = 128, BN = 64, KST = 2;
constexpr int TMEM_COLS = 256;              // of two blocks to an SM: S/P buffers [0,64) and [64,128), O [128,256)
constexpr float kRescaleThreshold = 8.f;    // log2 units
// One tcgen05.commit per MMA group, each completion signalled once and shared by all its waiters.  QK_DONE[s]: S of a tile
// of stage s is there (softmax) and K stage s is free (producer).  PV_DONE[s]: V stage s is free (producer), O includes
// tile j (rescale, epilogue; three blocks to an SM: P may be written again).
enum Bar {
  Q_FULL = 0, K_FULL0, K_FULL1, V_FULL0, V_FULL1, QK_DONE0, QK_DONE1, PV_DONE0, PV_DONE1,
  P_FULL0, P_FULL1, DRAIN, NUM_BARS
};
// self-test tile geometry (128 x 128 operands)
constexpr int TILE_BYTES = 128 * 128 * 2, SUB_BYTES = TILE_BYTES / 2;
}  // namespace tc

// Bounded wait that also gives up as soon as another role has aborted.  Small on purpose: it is inlined some
// twenty times into a kernel whose warps run different parts of the code at the same time.
__device__ __forceinline__ bool wait_or_abort(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  if (sm100::mbar_try_wait(bar, parity)) return true;
  const uint32_t t0 = static_cast<uint32_t>(clock());
#pragma unroll 1
  do {
    if (sm100::mbar_try_wait(bar, parity)) return true;
  } while (!*abort_flag && static_cast<uint32_t>(clock()) - t0 < static_cast<uint32_t>(sm100::kWaitLimitCycles));
  *abort_flag = 1;
  return false;
}

}  // namespace nvllm
