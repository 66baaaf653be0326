// Device side of the equal stretches of chains (ssd_chain_wrap): which item a block walks, and the hand-over of a chain's state to the block
// that walks the rest of it.
#pragma once
#include "ssd_fused.h"
#include "tc_common.cuh"

namespace pmb {

struct ChainItem { int chain, from, count; };            // in units of steps, in the order that the chain is walked in
// Round 0: the beginning of the chain that the stretch ends in; then its whole chains; then the rest of the chain that it begins in.
__device__ __forceinline__ ChainItem chain_item(const ChainWrap& w, int block, int units) {
  const int s = block % CHAIN_SMS, r = block / CHAIN_SMS;
  const ChainWrap::Entry& e = w.e[s];
  if (r == 0) return ChainItem{e.head, 0, e.head_units};
  if (r <= w.wholes) return ChainItem{w.first_whole + (r - 1) * CHAIN_SMS + s, 0, units};
  if (e.extra && r == w.wholes + 1) return ChainItem{e.extra, 0, units};
  return ChainItem{e.tail, e.tail_from, e.tail_from && r == w.wholes + (e.extra ? 2 : 1) ? units - e.tail_from : 0};
}

// Four warps of a block hand over, each after its own stores; four warps of another take.  The wait is bounded.
constexpr uint32_t HANDOVER_WARPS = 4, HANDOVER_LIMIT = 1u << 22;
__device__ __forceinline__ void chain_hand_over(uint32_t* flag) {
  __threadfence();
  __syncwarp();
  if ((threadIdx.x & 31) == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(flag) : "memory");
}
__device__ __forceinline__ bool chain_take(const uint32_t* flag, volatile uint32_t* abort_flag) {
  bool got = true;
  if ((threadIdx.x & 31) == 0) {
    got = false;
    for (uint32_t i = 0; i < HANDOVER_LIMIT && !got && !*abort_flag; ++i) {
      uint32_t v;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(flag) : "memory");
      got = v >= HANDOVER_WARPS;
      if (!got) __nanosleep(100);
    }
  }
  __syncwarp();
  __threadfence();
  return __all_sync(0xffffffffu, got);
}

}  // namespace pmb
