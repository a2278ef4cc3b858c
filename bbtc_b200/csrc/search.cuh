// Device searches shared by the per-task and the allocation-free count kernels.
#pragma once

#include <cstdint>

namespace bbtc {

__device__ __forceinline__ uint32_t lower_bound_u32(const uint32_t* a, uint32_t n, uint32_t x) {
  uint32_t lo = 0;
  while (n > 0) {
    const uint32_t half = n >> 1;
    if (a[lo + half] < x) {
      lo += half + 1;
      n -= half + 1;
    } else {
      n = half;
    }
  }
  return lo;
}

// First p in [from, n) with a[p] >= x (n if none) for a sorted a, given
// a[from - 1] < x: steps of 1, 2, 4, ... from `from`, then bisection of the
// last step.  A lane probing increasing ids of one row against a long pivot
// row moves forward from its previous position instead of bisecting the
// whole row again (skewed degrees: long pivot rows, short probe rows).
__device__ __forceinline__ uint32_t gallop_lb(const uint32_t* __restrict__ a, uint32_t n, uint32_t from, uint32_t x) {
  if (from >= n || a[from] >= x) return from;
  uint32_t lo = from, step = 1;  // a[lo] < x
  while (lo + step < n && a[lo + step] < x) {
    lo += step;
    step <<= 1;
  }
  uint32_t L = lo + 1;
  uint32_t len = min(lo + step, n) - L;  // the answer is in [L, L + len]
  while (len > 0) {
    const uint32_t half = len >> 1;
    if (a[L + half] < x) {
      L += half + 1;
      len -= half + 1;
    } else {
      len = half;
    }
  }
  return L;
}

// Row b holding entry e: the largest b with rp[b] <= e, a 32-way step at a
// time.  Stays below H whatever rp holds.
__device__ __forceinline__ uint32_t row_of(const uint32_t* __restrict__ rp, uint32_t H, uint32_t e) {
  const uint32_t lane = threadIdx.x & 31;
  uint32_t lo = 0, hi = H;
  while (hi - lo > 1) {
    const uint32_t step = (hi - lo + 31) / 32;
    const uint64_t at = lo + (uint64_t)(lane + 1) * step;
    const uint32_t below = __ballot_sync(0xffffffffu, at < hi && rp[at] <= e);
    lo += __popc(below) * step;
    hi = min(hi - lo, step) + lo;
  }
  return lo;
}

// Next row after b with an entry at or after e: 128 row ends a step.
__device__ __forceinline__ uint32_t next_row(const uint32_t* __restrict__ rp, uint32_t H, uint32_t b, uint32_t e,
                                             uint32_t lane) {
  b++;
  while (true) {
    uint32_t v[4];
#pragma unroll
    for (uint32_t q = 0; q < 4; q++) {
      const uint32_t idx = b + 32 * q + lane;
      v[q] = idx < H ? rp[idx + 1] : 0xffffffffu;
    }
#pragma unroll
    for (uint32_t q = 0; q < 4; q++) {
      const uint32_t mask = __ballot_sync(0xffffffffu, v[q] > e);
      if (mask) return b + 32 * q + __ffs(mask) - 1;
    }
    b += 128;
  }
}

}  // namespace bbtc
