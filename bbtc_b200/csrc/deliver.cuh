// The end of a queue kernel: its last warp hands the counts over.
//
// A count was four operations on its stream: clear the accumulators, the
// kernel, copy the counts back, wait.  With this it is the kernel and the
// wait, 4 to 5 us less (R-MAT s12: 37 -> 33 us a call).  Not inlined: its
// pointers would be live, in local memory, across the whole count (R-MAT s22
// 4.99 ms inlined, 4.92 as a call, 4.97 without it).  Adding the call made the
// fused kernel itself faster on small graphs (the same kernel without delivering
// through it: s16 82.6 us against 100 before, s18 200.6 against 230); why is not
// known, so a change of its code may take that back.
#pragma once
#include <cstdint>

namespace bbtc {

// outs: nouts counts, the control word (low half the queue head, high half
// the staging flag) and the number of warps that are done.  Called by every
// warp once, after its last addition (made by lane 0).  The last warp of the
// launch writes the counts and the control word to `host` (page-locked) and,
// unless NULL, `dev`, and leaves `outs` zero for the next launch.
static __device__ __noinline__ void deliver(unsigned long long* outs, uint32_t nouts, uint64_t* dev, uint64_t* host) {
  const uint32_t lane = threadIdx.x & 31;
  uint32_t before = 0;
  if (lane == 0) {
    __threadfence();  // this lane's additions come before its mark
    before = atomicAdd(reinterpret_cast<uint32_t*>(outs + nouts + 1), 1u);
  }
  before = __shfl_sync(0xffffffffu, before, 0);
  if (before + 1 != gridDim.x * (blockDim.x >> 5)) return;
  __threadfence();
  for (uint32_t i = lane; i < nouts + 2; i += 32) {
    const uint64_t v = __ldcg(outs + i);
    outs[i] = 0;
    if (i > nouts) continue;
    host[i] = v;
    if (dev) dev[i] = v;
  }
}

}  // namespace bbtc
