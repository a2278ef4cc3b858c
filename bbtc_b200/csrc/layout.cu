// Device-resident block-CSR layout.
//
// The reference splits the oriented CSR into P x P tile CSRs on the host:
// a per-row count by tile column, a serial exclusive scan over P*(N+P) row
// slots and a scatter of tile-local column ids
// (src/data_structures/block_csr.cpp:288-376), then copies tiles to the GPU
// lazily, one cudaMalloc + two copies + a stream sync per tile
// (src/triangle_counting/bb_tc_helper.cpp:75-110).  Here the whole layout is
// built on the device once and stays resident:
//
//   * the oriented CSR itself (global ids);
//   * its rows word-compressed: row u's ids grouped by 32-id word into (word
//     index, bit mask) pairs, which the fused count streams;
//   * the pivot lists of the fused count (internal.h: PivotGraph): the in-edges
//     (u, v) of every vertex v that has a row of its own, each with the range
//     of row u's pairs that can meet row v -- from the pair that holds v (or,
//     when row v has kept ids below v, from the first pair that can hold one:
//     see record_start) to the row's end.
//
// The P x P tiles of the per-task kernels are built on first use:
//
//   * forward tiles (x, y): rows of part x, tile-local columns of part y --
//     the reference's tiles, used as ab / bc / ac;
//   * reversed tiles (y, x): the same edges grouped by their column vertex --
//     the CSC of forward tile (x, y).
//
// Every tile owns a row-pointer segment of H+1 tile-local offsets (first
// entry 0) in one pool, laid out like the reference's rows_ array (P segments
// per row part); column segments hold only the non-empty tiles.  Segments
// start on 16-byte boundaries.  All passes are edge-parallel, so no thread
// walks a whole row.
#include <cub/cub.cuh>
#include <cuda.h>

#include <algorithm>
#include <cstring>

#include "internal.h"
#include "layout_check.hpp"
#include "search.cuh"

namespace bbtc {

namespace {

constexpr uint32_t FULLMASK = 0xffffffffu;

__device__ __forceinline__ uint32_t part_of(const uint32_t* cuts, uint32_t P, uint32_t u) {
  // largest x in [0, P) with cuts[x] <= u (skips empty parts); needs u < cuts[P]
  uint32_t lo = 0, hi = P;
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (cuts[mid] <= u) lo = mid; else hi = mid;
  }
  return lo;
}

// first position p in [lo, hi) with a[p] >= x
__device__ __forceinline__ uint32_t lower_bound_range(const uint32_t* __restrict__ a, uint32_t lo, uint32_t hi,
                                                      uint32_t x) {
  while (lo < hi) {
    const uint32_t mid = lo + ((hi - lo) >> 1);
    if (a[mid] < x) lo = mid + 1; else hi = mid;
  }
  return lo;
}

// Host-to-device copy done by the SMs: `src` is page-locked host memory
// mapped into the device's address space, read over the host link, so the
// copy does not queue behind other streams' transfers on the copy engines.
// Each `dst` is a device allocation (256-byte aligned); words = bytes / 4.
// Two arrays per launch (a graph's row pointers and ids); words1 may be 0.
__device__ __forceinline__ void copy_words(uint32_t* __restrict__ dst, const uint32_t* __restrict__ src,
                                           uint64_t words, uint64_t t0, uint64_t stride) {
  uint64_t done = 0;
  if ((reinterpret_cast<uintptr_t>(src) & 15) == 0) {
    const uint64_t v = words / 4;
    const uint4* __restrict__ s4 = reinterpret_cast<const uint4*>(src);
    uint4* __restrict__ d4 = reinterpret_cast<uint4*>(dst);
    for (uint64_t i = t0; i < v; i += stride) d4[i] = s4[i];
    done = v * 4;
  }
  for (uint64_t i = done + t0; i < words; i += stride) dst[i] = src[i];
}

__global__ void k_copy_mapped(uint32_t* __restrict__ dst0, const uint32_t* __restrict__ src0, uint64_t words0,
                              uint32_t* __restrict__ dst1, const uint32_t* __restrict__ src1, uint64_t words1) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  const uint64_t t0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  copy_words(dst0, src0, words0, t0, stride);
  copy_words(dst1, src1, words1, t0, stride);
}

// Cut vector of a launch, by value.
struct CutVec {
  uint32_t c[kMaxParts + 1];
  uint32_t P;
};

// Words of the flags block: what the build leaves for the host, and the tile
// tickets of the two single-pass kernels.
enum : uint32_t {
  kFlagBad = 0,
  kFlagUnoriented = 1,
  kFlagPivots = 2,
  kFlagPairs = 3,
  kFlagSparse = 4,
  kFlagTicketPairs = 5,
  kFlagTicketPivots = 6,
  kFlagWords = 8
};
constexpr uint32_t kBadWait = 1u << 30;  // in kFlagBad: a wait for an earlier tile ran out

// Row part of the input contract, a thread per row: row pointers start at 0,
// never decrease and end at m.  Sets the bit of every edge that starts a row
// in `heads`, and the unoriented flag when some row's first id does not exceed
// the row.
__global__ void k_row_heads(const uint32_t* __restrict__ indptr, const uint32_t* __restrict__ indices, uint32_t n,
                            uint64_t m, uint32_t* __restrict__ heads, uint32_t* __restrict__ flags) {
  for (uint64_t u = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; u < n; u += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t a = indptr[u], b = indptr[u + 1];
    if (u == 0 && a != 0) atomicOr(&flags[kFlagBad], 1u);
    if (u == n - 1 && (uint64_t)b != m) atomicOr(&flags[kFlagBad], 2u);
    if (b < a || (uint64_t)b > m) {
      atomicOr(&flags[kFlagBad], 4u);
    } else if (b > a) {
      atomicOr(&heads[a >> 5], 1u << (a & 31));
      if (indices[a] <= u) flags[kFlagUnoriented] = 1u;
    }
  }
}

// ---- single-pass tiles --------------------------------------------------------
// The two passes below number things (pairs, pivots) across the whole edge
// array in one read of it: a block takes the next tile by ticket, counts in
// it, publishes the count, and adds up the tiles before it from what they have
// published -- their own counts, or from some tile on the sum up to it.  A
// tile's word is (state << 62 | value): 0 nothing yet, 1 the tile's own, 2 up
// to and including it.  Tickets follow the order in which blocks start, so the
// tiles waited for are running or done; the waits are bounded all the same,
// and a block whose wait ran out leaves without writing (a sum that lacks
// tiles would send its writes out of range): the build fails.  With `dbg` > 0,
// the test hook of bbtc_debug_layout_timeout, the first tile publishes nothing
// and the waits give up after `dbg` polls.
// Tiles are small (8 warps of 8 chunks of 32) while few of them would leave
// SMs idle, and large (16 warps of 16 chunks) where the sum over earlier tiles
// would bound the pass.  Small and large, us: k_pairs R-MAT s12 7.2 / 12.4,
// s18 45 / 32, s22 570 / 420; k_pivots 8.8 / 16.9, 36 / 42, 371 / 276.  The large
// forms run at 40 registers (3 blocks of 16 warps an SM) and spill 40 and 148
// bytes a thread.
constexpr uint32_t kSmallWarps = 8, kSmallChunks = 8, kLargeWarps = 16, kLargeChunks = 16;
constexpr uint64_t kLargePairs = 1ull << 20, kLargePivots = 4ull << 20;  // edges from which tiles are large
inline uint64_t tile_size(bool large) {
  return 32 * (large ? (uint64_t)kLargeWarps * kLargeChunks : (uint64_t)kSmallWarps * kSmallChunks);
}
constexpr uint64_t kOwn = 1ull << 62, kUpTo = 2ull << 62;
constexpr uint32_t kTilePolls = 1u << 22;

__device__ __forceinline__ uint64_t tile_load(const uint64_t* p) {
  uint64_t v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void tile_store(uint64_t* p, uint64_t v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// What the tiles before tile i (in ticket order) hold together.  `a` carries
// counts; with HEADS, `b` carries for each tile the count from its first head
// on (0: no head) -- the counts run towards the tiles before, so the nearest
// tile with a head gives the count up to it.  Called by one warp; false when a
// tile has not published after `limit` polls, or another block gave up
// waiting: there is no sum then, and the block has to leave without using one.
struct TileSum {
  uint32_t count, head;
};
template <bool HEADS>
__device__ __forceinline__ bool tiles_before(const uint64_t* a, const uint64_t* b, uint32_t i, uint32_t* bad,
                                             uint32_t limit, TileSum& out) {
  const uint32_t lane = threadIdx.x & 31;
  out = TileSum{0, 0};
  uint32_t polls = 0;
  for (int64_t j = (int64_t)i - 1; j >= 0; j -= 32) {
    const int64_t at = j - lane;
    uint64_t va = kUpTo, vb = kUpTo;  // before the first tile: nothing
    bool ok, gave_up = false;
    do {
      if (at >= 0) {
        va = tile_load(a + at);
        vb = HEADS ? tile_load(b + at) : va;
      }
      ok = va >> 62 != 0 && va >> 62 == vb >> 62;  // both words of one publication
      if (!ok) gave_up = ++polls > limit || (polls % 1024 == 0 && (__ldcg(bad) & kBadWait));
    } while (!__all_sync(FULLMASK, ok || gave_up));
    if (!__all_sync(FULLMASK, ok)) {
      if (lane == 0) atomicOr(bad, kBadWait);
      return false;
    }
    const uint32_t sums = __ballot_sync(FULLMASK, va >> 62 == 2);
    const uint32_t last = sums ? __ffs(sums) - 1 : 32;  // the nearest tile with a sum
    const uint32_t own = lane < last ? (uint32_t)va : 0u;
    if (HEADS && out.head == 0) {
      const uint32_t some = __ballot_sync(FULLMASK, lane < last && (uint32_t)vb != 0);
      if (some) {  // the tiles between that head and here are in out.count and before it in the window
        const uint32_t f = __ffs(some) - 1;
        out.head = __shfl_sync(FULLMASK, (uint32_t)vb, f) + __reduce_add_sync(FULLMASK, lane > f ? own : 0u);
      } else if (last < 32) {
        out.head = __shfl_sync(FULLMASK, (uint32_t)vb, last);
        out.count += __reduce_add_sync(FULLMASK, own) + __shfl_sync(FULLMASK, (uint32_t)va, last);
        return true;
      }
    } else if (HEADS) {
      out.head += __reduce_add_sync(FULLMASK, own);
    }
    out.count += __reduce_add_sync(FULLMASK, own);
    if (last < 32) {
      const uint32_t sum = __shfl_sync(FULLMASK, (uint32_t)va, last);
      out.count += sum;
      if (HEADS && out.head) out.head += sum;
      return true;
    }
  }
  return true;
}

// Edge part of the input contract (rows strictly increasing, ids < n), the
// word-compressed rows and the records, in one read of the ids.  Pairs are
// numbered from the end of the array, pair p = m - (pairs opened from it on),
// so tiles run from the last edges to the first and the end of an edge's row
// -- the pair of the next row's first edge -- is known when the edge is
// reached.  A pair's edges are consecutive and their bits distinct, so its
// mask is a difference of running sums; the lane of the edge that opens it
// writes it.  head_pair[e] is written for edges that start a row.  Needs m > 0.
//
// It replaces a scan of the openings and a pass that read its result and
// searched the row ends: R-MAT s22 0.94 ms before, 0.42 now (1.3 GB moved: the
// shuffles and population counts of a chunk bound it, not memory), s12 20 us
// in three launches before, 7 in one.
template <uint32_t kTileWarps, uint32_t kTileChunks, int MINB>
__global__ void __launch_bounds__(32 * kTileWarps, MINB) k_pairs(const uint32_t* __restrict__ indices, const uint32_t* __restrict__ heads,
                                               uint32_t n, uint64_t m, uint2* __restrict__ words,
                                               uint2* __restrict__ rec, uint32_t* __restrict__ head_pair,
                                               uint64_t* __restrict__ sums, uint64_t* __restrict__ head_sums,
                                               uint32_t* __restrict__ flags, uint32_t dbg) {
  __shared__ uint32_t s_tile, s_summed, s_count[kTileWarps], s_head[kTileWarps];
  __shared__ TileSum s_before;
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr uint32_t kTile = kTileWarps * kTileChunks * 32;
  const uint32_t ntiles = (uint32_t)((m + kTile - 1) / kTile);
  while (true) {
    if (threadIdx.x == 0) s_tile = atomicAdd(&flags[kFlagTicketPairs], 1u);
    __syncthreads();
    const uint32_t i = s_tile;
    if (i >= ntiles) return;
    const uint64_t base = (uint64_t)(ntiles - 1 - i) * kTile + warp * (kTileChunks * 32);
    uint32_t x[kTileChunks];
#pragma unroll
    for (uint32_t c = 0; c < kTileChunks; c++) {
      const uint64_t e = base + 32 * c + lane;
      x[c] = e < m ? __ldg(indices + e) : 0u;
    }
    // lane c: the words of chunk c -- edges that start a row, edges that open a pair
    uint32_t my_heads = 0, my_opens = 0, bad = 0;
    if (lane < kTileChunks && base + 32 * lane < m) my_heads = __ldg(heads + (base >> 5) + lane);
    if (base == 0 && lane == 0) my_heads |= 1u;
    uint32_t before = base > 0 && base < m ? __ldg(indices + base - 1) : 0u;
#pragma unroll
    for (uint32_t c = 0; c < kTileChunks; c++) {
      const bool valid = base + 32 * c + lane < m;
      const bool head = (__shfl_sync(FULLMASK, my_heads, c) >> lane) & 1u;
      uint32_t prev = __shfl_up_sync(FULLMASK, x[c], 1);
      if (lane == 0) prev = before;
      before = __shfl_sync(FULLMASK, x[c], 31);
      if (valid && x[c] >= n) bad |= 8u;
      if (valid && !head && prev >= x[c]) bad |= 16u;
      const uint32_t o = __ballot_sync(FULLMASK, valid && (head || (prev ^ x[c]) >> 5 != 0));
      if (lane == c) my_opens = o;
    }
    if (bad) atomicOr(&flags[kFlagBad], bad);
    // the warp's pairs, and from its first head on
    const uint32_t count = __reduce_add_sync(FULLMASK, __popc(my_opens));
    {
      const uint32_t some = __ballot_sync(FULLMASK, my_heads != 0);
      uint32_t from = 0;
      if (some) {
        const uint32_t c = __ffs(some) - 1;
        from = __reduce_add_sync(FULLMASK, lane < c ? 0u
                                           : lane == c ? __popc(my_opens & (FULLMASK << (__ffs(my_heads) - 1)))
                                                       : __popc(my_opens));
      }
      if (lane == 0) {
        s_count[warp] = count;
        s_head[warp] = from;
      }
    }
    __syncthreads();
    // later warps of the tile, then the tiles before this one (they hold the later edges)
    uint32_t C = 0, H = 0, tile_C = 0, tile_H = 0;
    for (int w = kTileWarps - 1; w >= 0; w--) {
      if (w == (int)warp) {
        C = tile_C;
        H = tile_H;
      }
      if (s_head[w]) tile_H = tile_C + s_head[w];
      tile_C += s_count[w];
    }
    if (warp == 0) {
      if (lane == 0 && i > 0) {
        tile_store(sums + i, kOwn | tile_C);
        tile_store(head_sums + i, kOwn | tile_H);
      }
      TileSum b;
      const bool summed = tiles_before<true>(sums, head_sums, i, &flags[kFlagBad], dbg ? dbg : kTilePolls, b);
      if (lane == 0) s_summed = summed;
      if (lane == 0 && summed) {
        if (!dbg || i > 0) {
          tile_store(sums + i, kUpTo | (b.count + tile_C));
          tile_store(head_sums + i, kUpTo | (tile_H ? b.count + tile_H : b.head));
        }
        s_before = b;
        if (i == ntiles - 1) flags[kFlagPairs] = b.count + tile_C;
      }
    }
    __syncthreads();
    if (!s_summed) return;
    if (H) H += s_before.count; else H = s_before.head;
    C += s_before.count;
    // bits of the edges after the warp's that belong to its last pair
    uint32_t tail = 0;
    if (base + kTileChunks * 32 < m) {
      const uint64_t e = base + kTileChunks * 32 + lane;
      const uint32_t y = e < m ? __ldg(indices + e) : 0u;
      uint32_t prev = __shfl_up_sync(FULLMASK, y, 1);
      if (lane == 0) prev = before;
      const uint32_t hw = __ldg(heads + (e >> 5));
      const uint32_t o = __ballot_sync(FULLMASK, e >= m || ((hw >> lane) & 1u) || (prev ^ y) >> 5 != 0);
      const uint32_t f = o ? __ffs(o) - 1 : 32;
      tail = __reduce_or_sync(FULLMASK, lane < f ? 1u << (y & 31) : 0u);
    }
#pragma unroll
    for (int c = kTileChunks - 1; c >= 0; c--) {
      const uint64_t e = base + 32 * c + lane;
      const bool valid = e < m;
      const uint32_t o = __shfl_sync(FULLMASK, my_opens, c), hw = __shfl_sync(FULLMASK, my_heads, c);
      const uint32_t bit = valid ? 1u << (x[c] & 31) : 0u;
      uint32_t run = bit;  // running sum of the bits (modulo 2^32: only differences are used)
#pragma unroll
      for (uint32_t d = 1; d < 32; d <<= 1) {
        const uint32_t v = __shfl_up_sync(FULLMASK, run, d);
        if (lane >= d) run += v;
      }
      const uint32_t above = lane < 31 ? FULLMASK << (lane + 1) : 0u;
      const uint32_t next = o & above, next_head = hw & above;
      const uint32_t run_end = __shfl_sync(FULLMASK, run, next ? __ffs(next) - 2 : 31);
      const uint32_t p = (uint32_t)m - (C + __popc(next) + 1);
      if (valid) {
        const uint32_t end = next_head ? C + __popc(o & (FULLMASK << (__ffs(next_head) - 1))) : H;
        rec[e] = make_uint2(p, (uint32_t)m - end);
        if ((o >> lane) & 1u) {
          uint32_t mask = run_end - (run - bit);
          if (!next) mask |= tail;
          words[p] = make_uint2(x[c] >> 5, mask);
          if ((hw >> lane) & 1u) head_pair[e] = p;
        }
      }
      const uint32_t f = o ? __ffs(o) - 1 : 32;
      const uint32_t open_bits = __reduce_or_sync(FULLMASK, lane < f ? bit : 0u);
      tail = o ? open_bits : open_bits | tail;
      if (hw) H = C + __popc(o & (FULLMASK << (__ffs(hw) - 1)));
      C += __popc(o);
    }
    __syncthreads();
  }
}

// What the passes after the sort read.
struct PivotInput {
  const uint32_t* indptr;
  const uint32_t* indices;
  const uint32_t* head_pair;  // at every edge that starts a row: the row's first pair
  const uint32_t* keys;       // entries' vertices, sorted
  const uint2* words;
  uint32_t n;
  uint64_t m;
};

// First pair of row u (u <= n; an empty row's is its successor's).
__device__ __forceinline__ uint32_t row_pair(const PivotInput& in, uint32_t u) {
  const uint32_t e = in.indptr[u];
  return (uint64_t)e < in.m ? in.head_pair[e] : (uint32_t)in.m;
}

// Four consecutive batches of 32 entries with this many pivots or more count as sparse.
constexpr uint32_t kSparsePivots = 8;

// The pivots (8 words each, see PivotGraph), after the last one whose e0 is ~0,
// and crow, in one read of the sorted keys: a vertex is a pivot when it has
// in-edges and a row.  An entry whose key differs from the one before starts
// its vertex's in-edges and ends the previous vertex's.  It replaces four
// passes and five launches (R-MAT s22 0.32 ms, s12 23 us; now 0.28 ms and 9
// us).  (For a CSR with ids
// below their rows, k_fix_pivots and k_fix_entries go over the result.)
template <uint32_t kTileWarps, uint32_t kTileChunks, int MINB>
__global__ void __launch_bounds__(32 * kTileWarps, MINB) k_pivots(PivotInput in, uint32_t* __restrict__ piv, uint32_t* __restrict__ crow,
                                                uint64_t* __restrict__ sums, uint32_t* __restrict__ flags,
                                                uint32_t dbg) {
  if (flags[kFlagBad]) return;
  __shared__ uint32_t s_tile, s_summed, s_count[kTileWarps], s_before;
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint64_t m = in.m;
  constexpr uint32_t kTile = kTileWarps * kTileChunks * 32;
  const uint32_t ntiles = (uint32_t)((m + kTile - 1) / kTile);
  auto has_row = [&](uint32_t v) { return __ldg(in.indptr + v + 1) > __ldg(in.indptr + v); };
  while (true) {
    if (threadIdx.x == 0) s_tile = atomicAdd(&flags[kFlagTicketPivots], 1u);
    __syncthreads();
    const uint32_t i = s_tile;
    if (i >= ntiles) return;
    const uint64_t base = (uint64_t)i * kTile + warp * (kTileChunks * 32);
    uint32_t key[kTileChunks];
#pragma unroll
    for (uint32_t c = 0; c < kTileChunks; c++) {
      const uint64_t e = base + 32 * c + lane;
      key[c] = e < m ? __ldg(in.keys + e) : ~0u;
    }
    const uint32_t last_before = base > 0 && base < m ? __ldg(in.keys + base - 1) : ~0u;
    uint32_t start_bits = 0;  // bit c: this lane's entry of chunk c starts a vertex
    uint32_t r0[kTileChunks], r1[kTileChunks];  // and that vertex's row pointers, all asked for before any is looked at
#pragma unroll
    for (uint32_t c = 0; c < kTileChunks; c++) {
      uint32_t prev = __shfl_up_sync(FULLMASK, key[c], 1);
      const uint32_t left = c ? __shfl_sync(FULLMASK, key[c ? c - 1 : 0], 31) : last_before;
      if (lane == 0) prev = left;
      const bool start = base + 32 * c + lane < m && prev != key[c];
      start_bits |= start ? 1u << c : 0u;
      r0[c] = r1[c] = 0;
      if (start || (c == 0 && lane == 0 && base < m)) {
        r0[c] = __ldg(in.indptr + key[c]);
        r1[c] = __ldg(in.indptr + key[c] + 1);
      }
    }
    // lane c: of chunk c, the entries that start a vertex, those that start a
    // pivot, and whether its first entry's vertex is one
    uint32_t my_starts = 0, my_pivots = 0, my_first = 0;
    uint32_t row = 0;  // whether the vertex that is open has a row
#pragma unroll
    for (uint32_t c = 0; c < kTileChunks; c++) {
      const uint32_t starts = __ballot_sync(FULLMASK, (start_bits >> c) & 1u);
      uint32_t rows = 0;
      if (starts || c == 0) rows = __ballot_sync(FULLMASK, r1[c] > r0[c]);
      if (c == 0 || (starts & 1u)) row = rows & 1u;
      if (lane == c) {
        my_starts = starts;
        my_pivots = starts & rows;
        my_first = row;
      }
      if (starts) row = (rows >> (31 - __clz(starts))) & 1u;
    }
    const uint32_t mine = __popc(my_pivots);
    uint32_t incl = mine;
#pragma unroll
    for (uint32_t d = 1; d < 32; d <<= 1) {
      const uint32_t v = __shfl_up_sync(FULLMASK, incl, d);
      if (lane >= d) incl += v;
    }
    {
      const uint32_t ahead = __shfl_sync(FULLMASK, incl - mine, (lane + 4) & 31);
      const bool sparse = lane + 4 < kTileChunks && ahead - (incl - mine) >= kSparsePivots;
      const uint32_t some = __ballot_sync(FULLMASK, sparse);
      if (lane == 0 && some) atomicMax(&flags[kFlagSparse], (uint32_t)(base >> 5) + 35 - __clz(some));
    }
    if (lane == 31) s_count[warp] = incl;
    __syncthreads();
    uint32_t C = 0, tile_C = 0;
    for (uint32_t w = 0; w < kTileWarps; w++) {
      if (w == warp) C = tile_C;
      tile_C += s_count[w];
    }
    if (warp == 0) {
      if (lane == 0 && i > 0) tile_store(sums + i, kOwn | tile_C);
      TileSum b;
      const bool summed = tiles_before<false>(sums, sums, i, &flags[kFlagBad], dbg ? dbg : kTilePolls, b);
      if (lane == 0) s_summed = summed;
      if (lane == 0 && summed) {
        if (!dbg || i > 0) tile_store(sums + i, kUpTo | (b.count + tile_C));
        s_before = b.count;
        if (i == ntiles - 1) {
          const uint32_t k = b.count + tile_C;
          flags[kFlagPivots] = k;
          uint4* end = reinterpret_cast<uint4*>(piv + 8 * (uint64_t)k);
          end[0] = make_uint4(~0u, ~0u, 0, 0);
          end[1] = make_uint4(0, 0, 0, 0);
        }
      }
    }
    __syncthreads();
    if (!s_summed) return;
    C += s_before;
    if (lane < kTileChunks && base + 32 * lane < m)
      crow[(base >> 5) + lane] = C + (incl - mine) + (my_first ? (my_pivots & 1u) - 1u : 0u);
#pragma unroll
    for (uint32_t c = 0; c < kTileChunks; c++) {
      const uint32_t starts = __shfl_sync(FULLMASK, my_starts, c), pivots = __shfl_sync(FULLMASK, my_pivots, c);
      if (starts == 0) continue;
      const uint64_t e = base + 32 * c + lane;
      uint32_t prev = __shfl_up_sync(FULLMASK, key[c], 1);
      const uint32_t left = c ? __shfl_sync(FULLMASK, key[c ? c - 1 : 0], 31) : last_before;
      if (lane == 0) prev = left;
      if ((starts >> lane) & 1u) {
        const uint32_t k = C + __popc(pivots & ~(FULLMASK << lane));  // pivots before this entry
        if (e > 0 && has_row(prev)) piv[8 * (uint64_t)(k - 1) + 1] = (uint32_t)e;
        if ((pivots >> lane) & 1u) {
          const uint32_t v = key[c], a = __ldg(in.indptr + v), b = __ldg(in.indptr + v + 1);
          const uint32_t ws = in.head_pair[a], we = row_pair(in, v + 1);
          const uint32_t fw = __ldg(in.indices + a) >> 5, lw = __ldg(in.indices + b - 1) >> 5;
          uint32_t* d = piv + 8 * (uint64_t)k;
          d[0] = (uint32_t)e;
          *reinterpret_cast<uint2*>(d + 2) = make_uint2(ws, we - ws);
          *reinterpret_cast<uint4*>(d + 4) = make_uint4(fw, lw - fw + 1, FULLMASK, v);
        }
      }
      C += __popc(pivots);
    }
    // the warp of the last entry ends its vertex
    if (base < m && m <= base + kTileChunks * 32 && row && lane == 0) piv[8 * (uint64_t)(C - 1) + 1] = (uint32_t)m;
    __syncthreads();
  }
}

// ---- CSRs with ids below their rows -------------------------------------------
// The tasks (i, j, k) with j = part(v), i <= j <= k meet only in-edges of v
// from parts up to j (the entries are in source order) and ids of row v from
// cuts[j] on (the reference's tiles ab = (i, j), ac = (i, k), bc = (j, k),
// src/triangle_counting/gpu_sparse_kernel.cu:25-46).  Where every id exceeds
// its row's, that is all of them.

// The row that holds pair p.
__device__ uint32_t row_of_pair(const PivotInput& in, uint32_t p) {
  uint32_t lo = 0, hi = in.n;  // the last row whose first pair is <= p (empty rows share their successor's)
  while (hi - lo > 1) {
    const uint32_t mid = lo + ((hi - lo) >> 1);
    if (row_pair(in, mid) <= p) lo = mid; else hi = mid;
  }
  return lo;
}

__global__ void k_fix_pivots(PivotInput in, CutVec cuts, const uint2* __restrict__ rec, uint32_t npiv,
                             uint4* __restrict__ piv) {
  for (uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; k < npiv; k += (uint64_t)gridDim.x * blockDim.x) {
    uint4 d0 = piv[2 * k], d1 = piv[2 * k + 1];
    const uint32_t v = d1.w, part = part_of(cuts.c, cuts.P, v), row_end = in.indptr[v + 1];
    const uint32_t a = lower_bound_range(in.indices, in.indptr[v], row_end, cuts.c[part]);
    uint32_t lo = d0.x, hi = d0.y;  // first entry from a later part
    while (lo < hi) {
      const uint32_t mid = lo + ((hi - lo) >> 1);
      if (row_of_pair(in, rec[mid].x) < cuts.c[part + 1]) lo = mid + 1; else hi = mid;
    }
    d0.y = lo;
    if (a < row_end) {  // from the pair of the first kept id on
      const uint32_t fw = in.indices[a] >> 5, we = d0.z + d0.w;
      uint32_t p = d0.z, end = we;
      while (p < end) {
        const uint32_t mid = p + ((end - p) >> 1);
        if (in.words[mid].x < fw) p = mid + 1; else end = mid;
      }
      d0.z = p;
      d0.w = we - p;
      d1 = make_uint4(fw, (in.indices[row_end - 1] >> 5) - fw + 1, FULLMASK << (in.indices[a] & 31), v);
    } else {
      d0.z = d0.w = 0;
      d1 = make_uint4(0, 0, FULLMASK, v);
    }
    piv[2 * k] = d0;
    piv[2 * k + 1] = d1;
  }
}

// First pair of the record of entry (u, v): the streamed side is row u from
// the first pair whose word can hold a kept id of row v (first kept id L).
// When L lies in v's word or above that is the pair `p` holding v itself;
// otherwise the pair is searched in row u's pairs before p.
__device__ __forceinline__ uint32_t record_start(const PivotInput& in, uint32_t v, uint32_t lo, uint32_t p) {
  const uint32_t a = in.indptr[v], b = in.indptr[v + 1];
  const uint32_t k = lower_bound_range(in.indices, a, b, lo);
  if (k >= b) return p;  // no kept id
  const uint32_t lw = in.indices[k] >> 5;
  if (lw >= (v >> 5)) return p;
  uint32_t lo_p = row_pair(in, row_of_pair(in, p)), hi_p = p;  // the row holds v, so the answer is at or before p
  while (lo_p < hi_p) {
    const uint32_t mid = lo_p + ((hi_p - lo_p) >> 1);
    if (in.words[mid].x < lw) lo_p = mid + 1; else hi_p = mid;
  }
  return lo_p;
}

__global__ void k_fix_entries(PivotInput in, CutVec cuts, const uint4* __restrict__ piv, uint32_t* __restrict__ crow,
                              uint2* __restrict__ rec) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  const uint64_t t0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  for (uint64_t q = t0; 32 * q < in.m; q += stride) {
    const uint32_t k = crow[q];
    if (32 * q >= piv[2 * (uint64_t)k].y) crow[q] = k + 1;  // past the entries that it keeps
  }
  for (uint64_t q = t0; q < in.m; q += stride) {
    const uint32_t v = in.keys[q];
    rec[q].x = record_start(in, v, cuts.c[part_of(cuts.c, cuts.P, v)], rec[q].x);
  }
}

// Row id of every edge of a CSR that meets the contract.  A warp takes `run`
// consecutive edges (a multiple of 32), whatever their rows: it searches the
// first one's row in 32-way steps and then compares the edges with the ends of
// 32 rows at a time.  A warp per row left lanes idle (R-MAT s20, 15 edges a
// row: 90 us; now 52).
__global__ void k_row_ids(const uint32_t* __restrict__ indptr, uint32_t n, uint64_t m, uint32_t run,
                          uint32_t* __restrict__ rows) {
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t warps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  auto row_end = [&](uint32_t u) {  // of row u + lane; past the last row: above any edge
    return (uint64_t)u + lane < n ? __ldg(indptr + u + 1 + lane) : ~0u;
  };
  for (uint64_t c = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; c * run < m; c += warps) {
    const uint64_t end = min(m, (c + 1) * run);
    uint32_t u = row_of(indptr, n, (uint32_t)(c * run));
    uint32_t ends = row_end(u);
    for (uint64_t e0 = c * run; e0 < end; e0 += 32) {
      const uint64_t e = e0 + lane;
      bool done = e >= end;
      while (true) {
        uint32_t k = 0;  // rows of the window that end at or before e
#pragma unroll
        for (uint32_t step = 16; step > 0; step >>= 1)
          if (__shfl_sync(FULLMASK, ends, k + step - 1) <= e) k += step;
        const bool inside = __shfl_sync(FULLMASK, ends, k) > e;
        if (!done && inside) {
          rows[e] = u + k;
          done = true;
        }
        const uint32_t rest = __ballot_sync(FULLMASK, !done);
        if (!rest) break;
        const uint32_t next = (uint32_t)(e0 + __ffs(rest) - 1);
        u += 32;  // below n: a row past the window holds edge `next`
        ends = row_end(u);
        if (__shfl_sync(FULLMASK, ends, 31) <= next) {  // empty rows between, in any number
          u = row_of(indptr, n, next);
          ends = row_end(u);
        }
      }
    }
  }
}

// The parts of a cut vector in a block's shared memory.  An id's part: from the
// part of its bucket's first id on (part_of's bisection was most of the edge
// passes' instructions); a row's: from the part of a lower row on.
struct Parts {
  static constexpr uint32_t kBuckets = 1024;
  uint32_t cuts[kMaxParts + 1];
  uint32_t shift;
  uint8_t first[kBuckets];
  __device__ __forceinline__ void load(const uint32_t* __restrict__ g, uint32_t P) {
    for (uint32_t t = threadIdx.x; t <= P; t += blockDim.x) cuts[t] = g[t];
    const uint32_t ids = g[P], bits = 32 - __clz(ids);
    const uint32_t sh = bits > 10 ? bits - 10 : 0;  // ids < 2^bits: at most kBuckets buckets
    if (threadIdx.x == 0) shift = sh;
    __syncthreads();
    for (uint32_t b = threadIdx.x; b < kBuckets && (uint64_t)b << sh < ids; b += blockDim.x)
      first[b] = (uint8_t)part_of(cuts, P, b << sh);
    __syncthreads();
  }
  // `from`: the part of this id or of a lower one
  __device__ __forceinline__ uint32_t at(uint32_t id, uint32_t from) const {
    while (id >= cuts[from + 1]) from++;  // ends: id < cuts[P]
    return from;
  }
  __device__ __forceinline__ uint32_t of(uint32_t id) const { return at(id, first[id >> shift]); }
};

// Length of every (row, tile) run, added up in slot (rp_off[tile] + local row
// + 1) of the counts buffer, by the edges that start it or a batch of 32.  (The
// run's end was searched from its first edge: R-MAT s20, both directions, 180
// us; now 136, instructions bound it.)
__global__ void k_entry_count(const uint32_t* __restrict__ indices, const uint32_t* __restrict__ rows, uint64_t m,
                              const uint32_t* __restrict__ cuts_g, uint32_t P, const uint64_t* __restrict__ rp_off,
                              uint32_t* __restrict__ counts) {
  __shared__ Parts parts;
  parts.load(cuts_g, P);
  const uint32_t lane = threadIdx.x & 31;
  uint32_t x = 0;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t e0 = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) & ~31ull; e0 < m; e0 += stride) {
    const uint64_t e = e0 + lane;
    const uint32_t u = e < m ? rows[e] : ~0u;  // no row's number
    const uint32_t y = e < m ? parts.of(indices[e]) : 0u;
    const uint32_t pu = __shfl_up_sync(FULLMASK, u, 1), py = __shfl_up_sync(FULLMASK, y, 1);
    const bool first = lane == 0 || u != pu || y != py;
    const uint32_t later = __ballot_sync(FULLMASK, first) & (lane < 31 ? FULLMASK << (lane + 1) : 0u);
    if (first && e < m) {
      x = parts.at(u, x);
      atomicAdd(&counts[rp_off[x * P + y] + (u - parts.cuts[x]) + 1], (later ? __ffs(later) - 1 : 32u) - lane);
    }
  }
}

// Up to four zero fills of layout buffers in one launch, on the SMs (at the
// stream's priority, leaving the copy engines to the uploads); each range
// starts on a 16-byte boundary.
struct ZeroRanges {
  uint32_t* p[4];
  uint64_t words[4];
};

__global__ void k_zero_ranges(ZeroRanges z) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  const uint64_t t0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  for (int r = 0; r < 4; r++) {
    uint32_t* __restrict__ p = z.p[r];
    const uint64_t nwords = z.words[r];
    uint4* __restrict__ q = reinterpret_cast<uint4*>(p);
    const uint64_t n4 = nwords / 4;
    for (uint64_t i = t0; i < n4; i += stride) q[i] = make_uint4(0, 0, 0, 0);
    for (uint64_t i = n4 * 4 + t0; i < nwords; i += stride) p[i] = 0;
  }
}

// `scanned` is the inclusive scan of the run counts, so a slot minus its
// tile's first slot is the tile-local row pointer written to `rp`; per tile,
// the longest row and the number of non-empty rows (a row's length is the
// difference of two scanned slots).  blockIdx.y = tile: a pass over the pool
// as one array looked up every slot's tile (R-MAT s20, P 8: 63 us; now 21).
__global__ void k_localize_stats(uint32_t* __restrict__ rp, const uint32_t* __restrict__ scanned,
                                 const uint32_t* __restrict__ cuts, uint32_t P, const uint64_t* __restrict__ rp_off,
                                 uint32_t* __restrict__ maxdeg, uint32_t* __restrict__ nerows) {
  const uint32_t t = blockIdx.y, x = t / P;
  const uint32_t H = cuts[x + 1] - cuts[x];
  const uint64_t slots = ((uint64_t)H + 4) & ~3ull;  // H + 1 and the padding to the next tile
  if ((uint64_t)blockIdx.x * blockDim.x >= slots) return;
  __shared__ uint32_t longest, nonempty;
  if (threadIdx.x == 0) longest = nonempty = 0;
  __syncthreads();
  const uint64_t first = rp_off[t];
  const uint32_t base = scanned[first];
  uint32_t mx = 0, ne = 0;
  for (uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; r < slots; r += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t v = scanned[first + r];
    rp[first + r] = v - base;
    const uint32_t len = r < H ? scanned[first + r + 1] - v : 0u;
    mx = max(mx, len);
    ne += len != 0;
  }
  mx = __reduce_max_sync(FULLMASK, mx);
  ne = __reduce_add_sync(FULLMASK, ne);
  if ((threadIdx.x & 31) == 0 && ne) {
    atomicMax(&longest, mx);
    atomicAdd(&nonempty, ne);
  }
  __syncthreads();
  if (threadIdx.x == 0 && nonempty) {
    atomicMax(&maxdeg[t], longest);
    atomicAdd(&nerows[t], nonempty);
  }
}

// nnz per tile and 16-byte aligned column offsets of the non-empty tiles:
// one warp, 32 tiles at a time, an exclusive scan of the aligned sizes by
// shuffles (launched as one block of 32 threads).
__global__ void k_tile_offsets(const uint32_t* __restrict__ rp, const uint64_t* __restrict__ rp_off,
                               const uint32_t* __restrict__ cuts, uint32_t P, uint32_t* __restrict__ nnz,
                               uint64_t* __restrict__ col_off) {
  if (blockIdx.x != 0 || threadIdx.x >= 32) return;
  const uint32_t lane = threadIdx.x;
  const uint32_t T = P * P;
  uint64_t cur = 0;
  for (uint32_t t0 = 0; t0 < T; t0 += 32) {
    const uint32_t t = t0 + lane;
    uint32_t z = 0;
    if (t < T) {
      const uint32_t x = t / P;
      z = rp[rp_off[t] + (cuts[x + 1] - cuts[x])];
    }
    const uint64_t size = ((uint64_t)z + 3) & ~3ull;
    uint64_t incl = size;
#pragma unroll
    for (uint32_t d = 1; d < 32; d <<= 1) {
      const uint64_t o = __shfl_up_sync(FULLMASK, incl, d);
      if (lane >= d) incl += o;
    }
    if (t < T) {
      nnz[t] = z;
      col_off[t] = z ? cur + incl - size : kNoSegment;
    }
    cur += __shfl_sync(FULLMASK, incl, 31);
  }
}

// First edge of the (row, tile) run that holds edge `base` of row u, whose ids
// are `lo` or more: the first at or above (u, lo) in the edges' order.  Asked
// for by a whole warp: distances of 1, 2, 4, ... back from base, then 32-way
// steps.
__device__ __forceinline__ uint32_t run_start(const uint32_t* __restrict__ rows, const uint32_t* __restrict__ indices,
                                              uint32_t base, uint32_t u, uint32_t lo) {
  const uint32_t lane = threadIdx.x & 31;
  auto below = [&](uint64_t e) { return rows[e] < u || (rows[e] == u && indices[e] < lo); };
  const uint32_t before = __ballot_sync(FULLMASK, base < (1u << lane) || below(base - (1u << lane)));
  const uint32_t k = before ? __ffs(before) - 1 : 32;  // nearest distance 2^k that is before the run
  uint32_t hi = k == 0 ? base : base - (1u << (k - 1));
  uint32_t at = k == 32 || base < (1u << k) ? 0 : base - (1u << k) + 1;  // the answer is in [at, hi]
  while (at < hi) {
    const uint32_t step = (hi - at + 31) / 32;
    const uint64_t e = at + (uint64_t)lane * step;
    const uint32_t n = __popc(__ballot_sync(FULLMASK, e < hi && below(e)));
    if (n == 0) return at;
    hi = (uint32_t)min((uint64_t)hi, at + (uint64_t)n * step);
    at += (n - 1) * step + 1;
  }
  return at;
}

// Scatter tile-local column ids into the column pool, and the row index of
// every 32nd entry: erow[t][x / 32] = the row that holds entry x of tile t,
// for x = 0, 32, 64, ... < nnz, so that a work unit that starts at a multiple
// of 32 finds its first row with one load.  A warp takes kRunEdges consecutive
// edges.  Where a (row, tile) run starts among them its start is known; the run
// that they begin in is searched.  The edges of a run take its place in the
// pool from the first of them in the batch.  (The starts came from a max-scan
// over an array of all edges, the row index from a pass over the rows: R-MAT
// s20, both directions, 320 us; now 226.)
constexpr uint32_t kRunEdges = 128;
__global__ void k_entry_scatter(const uint32_t* __restrict__ indices, const uint32_t* __restrict__ rows, uint64_t m,
                                const uint32_t* __restrict__ cuts_g, uint32_t P, const uint64_t* __restrict__ rp_off,
                                const uint64_t* __restrict__ col_off, const uint32_t* __restrict__ rp,
                                uint32_t* __restrict__ col, uint32_t* __restrict__ erow) {
  __shared__ Parts parts;
  parts.load(cuts_g, P);
  const uint32_t* cuts = parts.cuts;
  const uint32_t lane = threadIdx.x & 31;
  uint32_t x = 0;
  const uint64_t warps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t w = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; w * kRunEdges < m; w += warps) {
    const uint32_t base = (uint32_t)(w * kRunEdges);
    uint32_t u[kRunEdges / 32], c[kRunEdges / 32];
#pragma unroll
    for (uint32_t k = 0; k < kRunEdges / 32; k++) {
      const uint64_t e = (uint64_t)base + 32 * k + lane;
      u[k] = e < m ? rows[e] : ~0u;  // no row's number
      c[k] = e < m ? indices[e] : 0u;
    }
    uint32_t run = 0, last_u = 0, last_y = 0;  // the run of the edges before these
#pragma unroll
    for (uint32_t k = 0; k < kRunEdges / 32; k++) {
      const uint32_t e0 = base + 32 * k, y = parts.of(c[k]);
      uint32_t pu = __shfl_up_sync(FULLMASK, u[k], 1), py = __shfl_up_sync(FULLMASK, y, 1);
      if (lane == 0) {
        pu = last_u;
        py = last_y;
      }
      last_u = __shfl_sync(FULLMASK, u[k], 31);
      last_y = __shfl_sync(FULLMASK, y, 31);
      bool first = u[k] != pu || y != py;
      if (k == 0) {
        run = run_start(rows, indices, base, __shfl_sync(FULLMASK, u[0], 0),
                        cuts[__shfl_sync(FULLMASK, y, 0)]);
        if (lane == 0) first = run == base;
      }
      const uint32_t starts = __ballot_sync(FULLMASK, first);
      // the first of each run's edges here looks the run's place up
      uint64_t tile_col = 0;
      uint32_t to = 0, index = 0, row = 0;
      if ((first || lane == 0) && u[k] != ~0u) {
        x = parts.at(u[k], x);
        const uint32_t t = x * P + y;
        row = u[k] - cuts[x];
        tile_col = col_off[t];
        index = (uint32_t)(tile_col / 32) + t;
        to = rp[rp_off[t] + row] - (first ? e0 + lane : run);  // modulo 2^32: plus an edge, its entry of the tile
      }
      const uint32_t mine = starts & (FULLMASK >> (31 - lane)), head = mine ? 31 - __clz(mine) : 0;
      tile_col = __shfl_sync(FULLMASK, tile_col, head);
      to = __shfl_sync(FULLMASK, to, head);
      index = __shfl_sync(FULLMASK, index, head);
      row = __shfl_sync(FULLMASK, row, head);
      if (u[k] != ~0u) {
        const uint32_t at = to + e0 + lane;
        col[tile_col + at] = c[k] - cuts[y];
        if ((at & 31) == 0) erow[index + (at >> 5)] = row;
      }
      if (starts) run = e0 + 31 - __clz(starts);
    }
  }
}

inline uint64_t align4(uint64_t x) { return (x + 3) & ~3ull; }

// True when [p, p + bytes) lies wholly inside one page-locked host allocation
// (or registered range) that the current device reads at the same address.
// Both ends are asked of the runtime, and the allocation's extent of the
// driver; any failure, or a driver that cannot answer, means "no".
bool mapped_host_range(const void* p, size_t bytes) {
  if (!p || bytes == 0 || (reinterpret_cast<uintptr_t>(p) & 3)) return false;
  const char* last = static_cast<const char*>(p) + bytes - 1;
  for (const void* q : {p, static_cast<const void*>(last)}) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, q) != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
    if (a.type != cudaMemoryTypeHost || a.devicePointer != q) return false;
  }
  using GetAttr = CUresult (*)(void*, CUpointer_attribute, CUdeviceptr);
  static const GetAttr get = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
    if (cudaGetDriverEntryPointByVersion("cuPointerGetAttribute", &f, 12000, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess) {
      cudaGetLastError();
      return static_cast<GetAttr>(nullptr);
    }
    return reinterpret_cast<GetAttr>(f);
  }();
  if (!get) return false;
  CUdeviceptr start = 0;
  size_t size = 0;
  if (get(&start, CU_POINTER_ATTRIBUTE_RANGE_START_ADDR, (CUdeviceptr)p) != CUDA_SUCCESS ||
      get(&size, CU_POINTER_ATTRIBUTE_RANGE_SIZE, (CUdeviceptr)p) != CUDA_SUCCESS)
    return false;
  const uint64_t b = (uint64_t)reinterpret_cast<uintptr_t>(p);
  return size > 0 && b >= start && b + bytes <= (uint64_t)start + size;
}

// Launch of a layout kernel.  A context with `open_carveout` (the server's
// large-request loaders) asks for the largest shared-memory carveout: an
// SM's split between L1 and shared memory changes only when the SM is idle,
// and a layout kernel (little shared memory of its own) otherwise runs with
// a small carveout, so while one of its blocks holds an SM -- a large
// graph's grid-stride pass runs a millisecond or more -- no block that needs
// more shared memory (a CUB scan or sort pass of a small request's layout, a
// count kernel) can start there, even from a higher-priority stream.  Other
// contexts keep the driver's choice, which leaves the passes their L1
// (R-MAT s22's layout is 2.8 ms slower with the largest carveout).
template <typename... KArgs, typename... Args>
int launch_layout(const bbtc_ctx* ctx, void (*kernel)(KArgs...), dim3 grid, dim3 block, cudaStream_t s,
                  Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = 0;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  if (ctx->open_carveout) {
    attr[0].id = cudaLaunchAttributePreferredSharedMemoryCarveout;
    attr[0].val.sharedMemCarveout = cudaSharedmemCarveoutMaxShared;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
  }
  BBTC_CUDA(cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...));
  return BBTC_OK;
}

// Build one block CSR (forward or reversed) from the edges' ids and row ids, in
// row order.  What the host keeps of it -- T column offsets
// (64-bit), then nnz, longest row and non-empty rows per tile -- lands in
// d_stats and, when the stream has run, in region `which` of the staging
// (read_stats).
int build_block(bbtc_ctx* ctx, BlockTiles& bt, const uint32_t* d_indices, const uint32_t* d_rows, uint64_t m,
                const std::vector<uint32_t>& cuts, const uint32_t* d_cuts, uint64_t* d_stats, int which, int grid) {
  const uint32_t P = (uint32_t)cuts.size() - 1;
  const uint32_t T = P * P;
  cudaStream_t s = ctx->stream;
  bt.P = P;
  bt.rp_off.assign(T, 0);
  uint64_t cur = 0;
  for (uint32_t x = 0; x < P; x++) {
    const uint64_t A = align4((uint64_t)cuts[x + 1] - cuts[x] + 1);
    for (uint32_t y = 0; y < P; y++) bt.rp_off[x * P + y] = cur + y * A;
    cur += A * P;
  }
  const uint64_t slots = cur;
  bt.rp_len = slots + 4;  // a 16-byte tail keeps rounded-up reads inside the pool
  bt.col_len = m + 4ull * T + 4;
  bt.erow_len = bt.col_len / 32 + T + 1;  // tile t's index starts at col_off[t] / 32 + t
  {
    cudaError_t e1 = dev_malloc(&bt.d_rp, bt.rp_len * sizeof(uint32_t), s);
    cudaError_t e2 = dev_malloc(&bt.d_col, bt.col_len * sizeof(uint32_t), s);
    cudaError_t e4 = dev_malloc(&bt.d_erow, bt.erow_len * sizeof(uint32_t), s);
    if (e1 != cudaSuccess || e2 != cudaSuccess || e4 != cudaSuccess) {
      cudaGetLastError();
      bt.release(s);
      return fail(BBTC_ERR_NOMEM, "device allocation of the block-CSR pools failed");
    }
  }
  bt.stream = s;
  DevBuf offs, counts;
  BBTC_TRY(dalloc(offs, T * sizeof(uint64_t), s));
  BBTC_TRY(dalloc(counts, bt.rp_len * sizeof(uint32_t), s));
  uint64_t* d_rp_off = offs.as<uint64_t>();
  {
    // through a pinned region that is not written again before the build's final sync
    char* h = ctx->h_stage + kStageOff[which];
    std::memcpy(h, bt.rp_off.data(), T * sizeof(uint64_t));
    BBTC_CUDA(cudaMemcpyAsync(d_rp_off, h, T * sizeof(uint64_t), cudaMemcpyHostToDevice, s));
  }
  uint64_t* d_coloff = d_stats;
  uint32_t* st_nnz = reinterpret_cast<uint32_t*>(d_stats + T);
  uint32_t* st_max = st_nnz + T;
  uint32_t* st_ne = st_nnz + 2 * T;
  {
    // run counts, column pool, tile statistics and the row-pointer pool's
    // 16-byte tail (every other slot of the pool is written below)
    ZeroRanges z{{counts.as<uint32_t>(), bt.d_col, reinterpret_cast<uint32_t*>(d_stats), bt.d_rp + slots},
                 {bt.rp_len, bt.col_len, 5ull * T, bt.rp_len - slots}};
    BBTC_TRY(launch_layout(ctx, k_zero_ranges, grid, 256, s, z));
  }
  if (m > 0)
    BBTC_TRY(launch_layout(ctx, k_entry_count, grid, 256, s, d_indices, d_rows, m, d_cuts, P, d_rp_off,
                           counts.as<uint32_t>()));
  // run counts -> their inclusive scan, in place: k_localize_stats turns it into tile-local row pointers
  {
    size_t tmp_bytes = 0;
    BBTC_CUDA(cub::DeviceScan::InclusiveSum(nullptr, tmp_bytes, counts.as<uint32_t>(), counts.as<uint32_t>(),
                                            (int64_t)slots, s));
    DevBuf tmp;
    BBTC_TRY(dalloc(tmp, tmp_bytes, s));
    BBTC_CUDA(cub::DeviceScan::InclusiveSum(tmp.p, tmp_bytes, counts.as<uint32_t>(), counts.as<uint32_t>(),
                                            (int64_t)slots, s));
  }
  uint32_t maxH = 1;
  for (uint32_t x = 0; x < P; x++) maxH = std::max(maxH, cuts[x + 1] - cuts[x]);
  const uint32_t blocks = std::min<uint32_t>(std::max(64u, 4096 / T), maxH / 1024 + 1);  // 4 slots a thread, or more
  BBTC_TRY(launch_layout(ctx, k_localize_stats, dim3(blocks, T), 256, s, bt.d_rp, counts.as<uint32_t>(), d_cuts, P,
                         d_rp_off, st_max, st_ne));
  BBTC_TRY(launch_layout(ctx, k_tile_offsets, 1, 32, s, bt.d_rp, d_rp_off, d_cuts, P, st_nnz, d_coloff));
  if (m > 0)
    BBTC_TRY(launch_layout(ctx, k_entry_scatter, grid, 256, s, d_indices, d_rows, m, d_cuts, P, d_rp_off,
                           d_coloff, bt.d_rp, bt.d_col, bt.d_erow));
  BBTC_CUDA(cudaMemcpyAsync(ctx->h_stage + kStageStats[which], d_stats, 20ull * T, cudaMemcpyDeviceToHost, s));
  return BBTC_OK;
}

// A built block CSR's statistics, from the staging (after the stream has run).
void read_stats(const bbtc_ctx* ctx, BlockTiles& bt, int which) {
  const uint32_t T = bt.P * bt.P;
  const uint64_t* hc = reinterpret_cast<const uint64_t*>(ctx->h_stage + kStageStats[which]);
  const uint32_t* hs = reinterpret_cast<const uint32_t*>(hc + T);
  bt.col_off.assign(hc, hc + T);
  bt.nnz.assign(hs, hs + T);
  bt.maxdeg.assign(hs + T, hs + 2 * T);
  bt.nerows.assign(hs + 2 * T, hs + 3 * T);
}

// Layout kernels are grid-stride loops: no more blocks than the largest array
// needs (a tiny graph's layout leaves the GPU to others), at most the
// context's cap.
int layout_grid(const bbtc_ctx* ctx, uint32_t n, uint64_t m, uint32_t P) {
  const uint64_t span = std::max<uint64_t>(m, (uint64_t)P * ((uint64_t)n + P));
  return (int)std::min<uint64_t>((uint64_t)ctx->sms * ctx->layout_blocks_per_sm,
                                 std::max<uint64_t>(ctx->sms, (span + 2047) / 2048));
}

uint64_t block_bytes(const BlockTiles& t) { return (t.rp_len + t.col_len + t.erow_len) * sizeof(uint32_t); }

int key_bits(uint64_t n) {
  int b = 1;
  while (b < 32 && (1ull << b) < n) b++;
  return b;
}

}  // namespace

void BlockTiles::release(cudaStream_t s) {
  if (d_rp) cudaFreeAsync(d_rp, s);
  if (d_col) cudaFreeAsync(d_col, s);
  if (d_erow) cudaFreeAsync(d_erow, s);
  d_rp = d_col = d_erow = nullptr;
}

DevTile dev_tile(const BlockTiles& t, const std::vector<uint32_t>& cuts, uint32_t x, uint32_t y) {
  DevTile d{};
  const uint32_t id = x * t.P + y;
  d.H = cuts[x + 1] - cuts[x];
  d.W = cuts[y + 1] - cuts[y];
  d.nnz = t.nnz[id];
  d.maxdeg = t.maxdeg[id];
  if (d.nnz) {
    d.rp = t.d_rp + t.rp_off[id];
    d.col = t.d_col + t.col_off[id];
    d.erow = t.d_erow + t.col_off[id] / 32 + id;
  } else {
    d.rp = d.col = d.erow = nullptr;
  }
  return d;
}

// Layout scratch a context keeps between builds: the temporaries of a graph
// of up to about nine million edges (about 28 bytes per edge); a larger
// build allocates its own and frees them at its end.
constexpr size_t kScratchKeep = 256ull << 20;

// Makes the context's kept scratch the running build's for the scope's
// lifetime, then grows the kept block to what the build asked for (a quarter
// more, at most kScratchKeep).  The kept block is a cache: when growing it
// fails the next build allocates as before, so it bypasses the allocation
// fault hook.  Its old block is freed behind the build's work on the stream.
struct ScratchScope {
  bbtc_ctx* ctx;
  cudaStream_t s;
  Scratch arena;
  Scratch* prev;
  ScratchScope(bbtc_ctx* c, cudaStream_t st) : ctx(c), s(st), prev(t_scratch) {
    arena.base = c->d_scratch;
    arena.cap = c->scratch_cap;
    t_scratch = &arena;
  }
  ~ScratchScope() {
    t_scratch = prev;
    if (arena.want <= ctx->scratch_cap || arena.want > kScratchKeep) return;
    if (ctx->d_scratch) cudaFreeAsync(ctx->d_scratch, s);
    ctx->d_scratch = nullptr;
    ctx->scratch_cap = 0;
    const size_t cap = std::min(kScratchKeep, ((arena.want + arena.want / 4) + (1u << 20) - 1) & ~size_t((1u << 20) - 1));
    void* p = nullptr;
    if (cudaMallocAsync(&p, cap, s) == cudaSuccess) {
      ctx->d_scratch = static_cast<char*>(p);
      ctx->scratch_cap = cap;
    } else {
      cudaGetLastError();
    }
  }
  ScratchScope(const ScratchScope&) = delete;
  ScratchScope& operator=(const ScratchScope&) = delete;
};

int build_layout(bbtc_graph* g, const uint32_t* in_indptr, const uint32_t* in_indices, bool host) {
  Range range("bbtc upload + layout");
  bbtc_ctx* ctx = g->ctx;
  cudaStream_t s = ctx->stream;
  ScratchScope scratch(ctx, s);
  const uint32_t n = g->n;
  const uint64_t m = g->m;
  const int grid = layout_grid(ctx, n, m, 1);
  for (cudaEvent_t& ev : ctx->ev_layout)
    if (!ev) BBTC_CUDA(cudaEventCreate(&ev));
  BBTC_CUDA(cudaEventRecord(ctx->ev_layout[0], s));

  const uint64_t mm = std::max<uint64_t>(m, 1);
  const uint64_t npiv_max = std::min<uint64_t>(n, m);
  g->nentry_rows = mm / 32 + 1;
  {
    cudaError_t e1 = dev_malloc(&g->d_words, mm * sizeof(uint2), s);
    cudaError_t e2 = dev_malloc(&g->d_rec, mm * sizeof(uint2), s);
    cudaError_t e3 = dev_malloc(&g->d_piv, (npiv_max + 1) * 2 * sizeof(uint4), s);
    cudaError_t e4 = dev_malloc(&g->d_crow, g->nentry_rows * sizeof(uint32_t), s);
    if (e1 != cudaSuccess || e2 != cudaSuccess || e3 != cudaSuccess || e4 != cudaSuccess) {
      cudaGetLastError();
      return fail(BBTC_ERR_NOMEM, "device allocation of the word-compressed rows and pivot lists failed");
    }
  }
  // The flags, the row heads and the tiles' words start at zero; the flags are
  // read back once, at the end: every pass between stays inside its arrays
  // whatever the input, or returns at once when the contract flag is set.
  // Allocated and cleared before the upload is queued, which the upload then
  // hides.
  const bool large_pairs = m >= kLargePairs, large_pivots = m >= kLargePivots;
  const uint64_t pair_tiles = (mm + tile_size(large_pairs) - 1) / tile_size(large_pairs);
  const uint64_t pivot_tiles = (mm + tile_size(large_pivots) - 1) / tile_size(large_pivots);
  const uint64_t hw = (mm / 32 + 4) & ~3ull;
  const uint64_t zero_words = kFlagWords + hw + 2 * (2 * pair_tiles + pivot_tiles);
  DevBuf zeroed;
  BBTC_TRY(dalloc(zeroed, zero_words * sizeof(uint32_t), s));
  uint32_t* flags = zeroed.as<uint32_t>();
  uint32_t* heads = flags + kFlagWords;
  uint64_t* sums = reinterpret_cast<uint64_t*>(heads + hw);
  {
    ZeroRanges z{{flags, reinterpret_cast<uint32_t*>(g->d_count), nullptr, nullptr}, {zero_words, 2 * kCountWords, 0, 0}};
    BBTC_TRY(launch_layout(ctx, k_zero_ranges, (int)std::min<uint64_t>((uint64_t)grid, zero_words / 1024 + 1), 256, s, z));
  }
  // the graph keeps its own copy of the oriented CSR
  {
    cudaError_t e1 = dev_malloc(&g->d_indptr, ((size_t)n + 1) * sizeof(uint32_t), s);
    cudaError_t e2 = dev_malloc(&g->d_indices, std::max<uint64_t>(m, 1) * sizeof(uint32_t) + 16, s);
    if (e1 != cudaSuccess || e2 != cudaSuccess) {
      cudaGetLastError();
      return fail(BBTC_ERR_NOMEM, "device allocation of the CSR copy failed");
    }
    const cudaMemcpyKind kind = host ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToDevice;
    // host copies in 8 MiB pieces: a copy engine runs one copy at a time, and
    // another stream's small upload then waits behind one piece, not behind
    // a whole large graph (273 MB at R-MAT s22: about 5 ms)
    // With an upload window (the server's large requests) at most that many
    // pieces are queued at once, so the copy engines' queues never hold a
    // large graph's whole upload ahead of another stream's small one.
    const uint32_t window = host ? ctx->upload_window : 0;
    cudaEvent_t evs[8] = {};
    struct EvRing {
      cudaEvent_t* e;
      ~EvRing() {
        for (int i = 0; i < 8; i++)
          if (e[i]) cudaEventDestroy(e[i]);
      }
    } ring{evs};
    uint32_t issued = 0;
    uint32_t by_kernel = 0;
    auto mapped = [&](const void* src, size_t bytes) {
      return host && bytes <= ctx->zero_copy_bytes && mapped_host_range(src, bytes);
    };
    // arrays that the SMs read over the host link, copied by one kernel launch
    uint32_t* kdst[2] = {nullptr, nullptr};
    const uint32_t* ksrc[2] = {nullptr, nullptr};
    uint64_t kwords[2] = {0, 0};
    auto copy = [&](void* dst, const void* src, size_t bytes) -> int {
      if (mapped(src, bytes)) {
        kdst[by_kernel] = static_cast<uint32_t*>(dst);
        ksrc[by_kernel] = static_cast<const uint32_t*>(src);
        kwords[by_kernel] = bytes / 4;
        by_kernel++;
        return BBTC_OK;
      }
      const size_t piece = host ? (size_t)8 << 20 : bytes;
      for (size_t o = 0; o < bytes; o += piece) {
        if (window) {
          cudaEvent_t& ev = evs[issued % std::min<uint32_t>(window, 8)];
          if (ev) BBTC_CUDA(cudaEventSynchronize(ev));
          else BBTC_CUDA(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
        }
        BBTC_CUDA(cudaMemcpyAsync(static_cast<char*>(dst) + o, static_cast<const char*>(src) + o,
                                  std::min(piece, bytes - o), kind, s));
        if (window) BBTC_CUDA(cudaEventRecord(evs[issued % std::min<uint32_t>(window, 8)], s));
        issued++;
      }
      return BBTC_OK;
    };
    BBTC_TRY(copy(g->d_indptr, in_indptr, ((size_t)n + 1) * sizeof(uint32_t)));
    if (m) BBTC_TRY(copy(g->d_indices, in_indices, m * sizeof(uint32_t)));
    if (by_kernel) {
      const uint64_t words = std::max(kwords[0], kwords[1]);
      const uint64_t blocks = std::max<uint64_t>(1, (words + 4095) / 4096);
      BBTC_TRY(launch_layout(ctx, k_copy_mapped, (int)std::min<uint64_t>(blocks, 2ull * ctx->sms), 256, s, kdst[0],
                             ksrc[0], kwords[0], kdst[1], ksrc[1], kwords[1]));
    }
    g->zero_copy = by_kernel > 0;
  }
  const uint32_t* d_indptr = g->d_indptr;
  const uint32_t* d_indices = g->d_indices;

  DevBuf rec_in, keys, head_pair;
  BBTC_TRY(dalloc(rec_in, mm * sizeof(uint2), s));
  BBTC_TRY(dalloc(keys, mm * sizeof(uint32_t), s));
  BBTC_TRY(dalloc(head_pair, mm * sizeof(uint32_t), s));
  if (n > 0) {
    BBTC_TRY(launch_layout(ctx, k_row_heads, grid, 256, s, d_indptr, d_indices, n, m, heads, flags));
  } else if (m > 0) {
    BBTC_CUDA(cudaMemsetAsync(flags, 0xff, sizeof(uint32_t), s));  // edges without rows
  }
  const PivotInput in{d_indptr,           d_indices, head_pair.as<uint32_t>(), keys.as<uint32_t>(),
                      static_cast<uint2*>(g->d_words), n, m};
  uint2* rec = static_cast<uint2*>(g->d_rec);
  if (n > 0 && m > 0) {
    auto tile_grid = [&](uint64_t tiles) { return (int)std::min<uint64_t>(tiles, (uint64_t)grid); };
    BBTC_TRY(launch_layout(ctx,
                           large_pairs ? k_pairs<kLargeWarps, kLargeChunks, 3> : k_pairs<kSmallWarps, kSmallChunks, 4>,
                           tile_grid(pair_tiles), 32 * (large_pairs ? kLargeWarps : kSmallWarps), s, d_indices, heads, n,
                           m, static_cast<uint2*>(g->d_words), rec_in.as<uint2>(), head_pair.as<uint32_t>(), sums,
                           sums + pair_tiles, flags, ctx->debug_layout_pass == 1 ? ctx->debug_layout_polls : 0u));
    // a stable sort of the records by column keeps every in-list in source order
    size_t tb = 0;
    BBTC_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tb, d_indices, keys.as<uint32_t>(), rec_in.as<uint2>(), rec,
                                              (int64_t)m, 0, key_bits(n), s));
    DevBuf tmp;
    BBTC_TRY(dalloc(tmp, tb, s));
    BBTC_CUDA(cub::DeviceRadixSort::SortPairs(tmp.p, tb, d_indices, keys.as<uint32_t>(), rec_in.as<uint2>(), rec,
                                              (int64_t)m, 0, key_bits(n), s));
    BBTC_TRY(launch_layout(
        ctx, large_pivots ? k_pivots<kLargeWarps, kLargeChunks, 3> : k_pivots<kSmallWarps, kSmallChunks, 4>,
        tile_grid(pivot_tiles), 32 * (large_pivots ? kLargeWarps : kSmallWarps), s, in, static_cast<uint32_t*>(g->d_piv),
        g->d_crow, sums + 2 * pair_tiles, flags, ctx->debug_layout_pass == 2 ? ctx->debug_layout_polls : 0u));
  }
  uint32_t* h = reinterpret_cast<uint32_t*>(ctx->h_stage + kStageFlags);
  BBTC_CUDA(cudaMemcpyAsync(h, flags, kFlagWords * sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
  BBTC_CUDA(cudaEventRecord(ctx->ev_layout[1], s));
  BBTC_CUDA(cudaStreamSynchronize(s));
  const uint32_t bad = h[kFlagBad];
  if (bad != 0xffffffffu && (bad & kBadWait))
    return fail(BBTC_ERR_TIMEOUT, "a layout pass waited too long for an earlier tile");
  if (bad) {
    std::string why;
    if (bad == 0xffffffffu) why += " edges but no rows;";
    else {
      if (bad & 1) why += " indptr[0] != 0;";
      if (bad & 2) why += " indptr[n] != m;";
      if (bad & 4) why += " row pointers decrease or exceed m;";
      if (bad & 8) why += " a column id >= n;";
      if (bad & 16) why += " a row is not strictly increasing (unsorted or duplicate ids);";
    }
    return fail(BBTC_ERR_INPUT, "CSR breaks the input contract:" + why);
  }
  g->oriented = h[kFlagUnoriented] == 0;
  g->npiv = h[kFlagPivots];
  g->nwords = h[kFlagPairs];
  g->sparse_end = h[kFlagSparse];
  if (!g->oriented && m > 0) {
    CutVec cuts{};
    std::copy(g->cuts.begin(), g->cuts.end(), cuts.c);
    cuts.P = g->P;
    uint4* piv = static_cast<uint4*>(g->d_piv);
    BBTC_TRY(launch_layout(ctx, k_fix_pivots, grid, 256, s, in, cuts, rec, g->npiv, piv));
    BBTC_TRY(launch_layout(ctx, k_fix_entries, grid, 256, s, in, cuts, piv, g->d_crow, rec));
    BBTC_CUDA(cudaEventRecord(ctx->ev_layout[1], s));
    BBTC_CUDA(cudaStreamSynchronize(s));
  }
  float ms = 0;
  BBTC_CUDA(cudaEventElapsedTime(&ms, ctx->ev_layout[0], ctx->ev_layout[1]));
  g->layout_ms = ms;
  g->device_bytes = ((uint64_t)n + 1 + m + g->nentry_rows) * sizeof(uint32_t) + 64 * sizeof(uint64_t) +
                    2 * mm * sizeof(uint2) + (npiv_max + 1) * 2 * sizeof(uint4);
  return BBTC_OK;
}

namespace {

// Block CSRs of the per-task kernels, from the resident CSR (which passed the
// contract check when it was uploaded): the forward one, the reversed one from
// the edges sorted by column (stable, so in-lists stay in source order), or
// both, which share the row ids and one wait.  The first per-task count of a
// graph pays for them (R-MAT s12 / s18 / s20, cuts into 8 equal parts, half the
// list, us: 188 / 378 / 1,011, the next count 34 / 19 / 18; built apart, each
// with its own row ids and wait, 249 / 528 / 1,434).
int build_tiles(bbtc_graph* g, bool forward, bool reversed) {
  Range range("bbtc block CSRs");
  bbtc_ctx* ctx = g->ctx;
  cudaStream_t s = ctx->stream;
  BBTC_CUDA(cudaSetDevice(ctx->device));
  ScratchScope scratch(ctx, s);
  const uint32_t n = g->n, P = g->P, T = P * P;
  const uint64_t m = g->m, mm = std::max<uint64_t>(m, 1);
  const int grid = layout_grid(ctx, n, m, P);
  DevBuf d_cuts, rows, stats[2], keys, sources;
  BBTC_TRY(dalloc(d_cuts, g->cuts.size() * sizeof(uint32_t), s));
  BBTC_TRY(dalloc(rows, mm * sizeof(uint32_t), s));
  {
    uint32_t* h = reinterpret_cast<uint32_t*>(ctx->h_stage + kStageCuts);
    std::memcpy(h, g->cuts.data(), g->cuts.size() * sizeof(uint32_t));
    BBTC_CUDA(cudaMemcpyAsync(d_cuts.p, h, g->cuts.size() * sizeof(uint32_t), cudaMemcpyHostToDevice, s));
  }
  if (m > 0) {  // an even share of the edges per warp, but few where they are few
    const uint64_t share = (m + 8ull * grid - 1) / (8ull * grid);
    const uint32_t run = (uint32_t)std::min<uint64_t>(std::max<uint64_t>((share + 31) & ~31ull, 64), 4096);
    BBTC_TRY(launch_layout(ctx, k_row_ids, grid, 256, s, g->d_indptr, n, m, run, rows.as<uint32_t>()));
  }
  if (forward) {
    BBTC_TRY(dalloc(stats[0], 20ull * T, s));
    BBTC_TRY(build_block(ctx, g->fwd, g->d_indices, rows.as<uint32_t>(), m, g->cuts,
                         d_cuts.as<uint32_t>(), stats[0].as<uint64_t>(), 0, grid));
  }
  if (reversed) {
    BBTC_TRY(dalloc(keys, mm * sizeof(uint32_t), s));
    BBTC_TRY(dalloc(sources, mm * sizeof(uint32_t), s));
    if (m > 0) {
      size_t tb = 0;
      BBTC_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tb, g->d_indices, keys.as<uint32_t>(), rows.as<uint32_t>(),
                                                sources.as<uint32_t>(), (int64_t)m, 0, key_bits(n), s));
      DevBuf tmp;
      BBTC_TRY(dalloc(tmp, tb, s));
      BBTC_CUDA(cub::DeviceRadixSort::SortPairs(tmp.p, tb, g->d_indices, keys.as<uint32_t>(), rows.as<uint32_t>(),
                                                sources.as<uint32_t>(), (int64_t)m, 0, key_bits(n), s));
    }
    BBTC_TRY(dalloc(stats[1], 20ull * T, s));
    BBTC_TRY(build_block(ctx, g->rev, sources.as<uint32_t>(), keys.as<uint32_t>(), m, g->cuts,
                         d_cuts.as<uint32_t>(), stats[1].as<uint64_t>(), 1, grid));
  }
  BBTC_CUDA(cudaStreamSynchronize(s));
  if (forward) {
    read_stats(ctx, g->fwd, 0);
    g->fwd_built = true;
    g->device_bytes += block_bytes(g->fwd);
  }
  if (reversed) {
    read_stats(ctx, g->rev, 1);
    g->rev_built = true;
    g->device_bytes += block_bytes(g->rev);
  }
  return BBTC_OK;
}

int ensure(bbtc_graph* g, bool forward, bool reversed) {
  forward = forward && !g->fwd_built;
  reversed = reversed && !g->rev_built;
  if (!forward && !reversed) return BBTC_OK;
  const int rc = build_tiles(g, forward, reversed);
  if (rc != BBTC_OK) {
    // a failed build (say, out of memory half way) leaves nothing behind: the
    // frees are stream-ordered after whatever of it was enqueued
    for (BlockTiles* bt : {forward ? &g->fwd : nullptr, reversed ? &g->rev : nullptr})
      if (bt) {
        bt->release(g->ctx->stream);
        *bt = BlockTiles();
      }
  }
  return rc;
}

}  // namespace

int ensure_fwd(bbtc_graph* g) { return ensure(g, true, false); }

int ensure_tiles(bbtc_graph* g) { return ensure(g, true, true); }

}  // namespace bbtc

// Read the whole layout back and check it on the host (debug aid: it copies
// every array, so it costs about the graph's device bytes in host memory and
// PCIe time).  The block CSRs of the per-task kernels are checked when they have been built.
int bbtc_graph_validate(const bbtc_graph* g) {
  using namespace bbtc;
  static_assert(check::kNoSeg == kNoSegment, "empty-tile marker");
  if (!g) return fail(BBTC_ERR_ARG, "NULL graph");
  bbtc_ctx* ctx = g->ctx;
  Range range("bbtc validate");
  cudaStream_t s = ctx->stream;
  BBTC_CUDA(cudaSetDevice(ctx->device));
  const uint32_t n = g->n;
  const uint64_t m = g->m;
  const uint64_t mm = std::max<uint64_t>(m, 1);
  auto get = [&](std::vector<uint32_t>& h, const void* d, uint64_t words) -> int {
    h.assign(words, 0);
    if (words) BBTC_CUDA(cudaMemcpyAsync(h.data(), d, words * sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
    return BBTC_OK;
  };
  std::vector<uint32_t> indptr, indices, pairs, rec, piv, crow;
  BBTC_TRY(get(indptr, g->d_indptr, (uint64_t)n + 1));
  BBTC_TRY(get(indices, g->d_indices, mm));
  const uint32_t at = (uint32_t)(m - g->nwords);  // pairs sit at their array's end
  BBTC_TRY(get(pairs, static_cast<const uint2*>(g->d_words) + at, 2 * g->nwords));
  BBTC_TRY(get(rec, g->d_rec, 2 * m));
  BBTC_TRY(get(piv, g->d_piv, m ? 8 * ((uint64_t)g->npiv + 1) : 0));
  BBTC_TRY(get(crow, g->d_crow, (m + 31) / 32));
  BBTC_CUDA(cudaStreamSynchronize(s));
  for (uint32_t& p : rec) p -= at;
  for (uint32_t k = 0; m && k < g->npiv; k++)
    if (piv[8 * (uint64_t)k + 3]) piv[8 * (uint64_t)k + 2] -= at;
  check::Csr c{n, m, indptr.data(), indices.data()};
  std::string why = check::csr(c);
  std::vector<uint32_t> wptr((size_t)n + 1, 0), tp, tc;
  check::Words w{wptr.data(), pairs.data(), g->nwords};
  if (why.empty()) {
    check::row_pairs(c, wptr.data());
    why = check::words(c, w);
  }
  if (why.empty()) check::transpose(c, tp, tc);
  const check::Csr tr{n, m, tp.data(), tc.data()};
  if (why.empty() && m)
    why = check::pivots(c, tr, w, check::Pivots{g->P, g->cuts.data(), g->npiv, piv.data(), rec.data(), crow.data()});
  for (int pass = 0; pass < 2 && why.empty(); pass++) {
    const BlockTiles& bt = pass == 0 ? g->rev : g->fwd;
    if (!(pass == 0 ? g->rev_built : g->fwd_built)) continue;
    std::vector<uint32_t> rp, col, erow;
    BBTC_TRY(get(rp, bt.d_rp, bt.rp_len));
    BBTC_TRY(get(col, bt.d_col, bt.col_len));
    BBTC_TRY(get(erow, bt.d_erow, bt.erow_len));
    BBTC_CUDA(cudaStreamSynchronize(s));
    check::Tiles t;
    t.P = g->P;
    t.cuts = g->cuts.data();
    t.rp_off = bt.rp_off.data();
    t.col_off = bt.col_off.data();
    t.nnz = bt.nnz.data();
    t.maxdeg = bt.maxdeg.data();
    t.nerows = bt.nerows.data();
    t.rp = rp.data();
    t.rp_len = bt.rp_len;
    t.col = col.data();
    t.col_len = bt.col_len;
    t.erow = erow.data();
    t.erow_len = bt.erow_len;
    why = check::tiles(pass == 0 ? "reversed tiles" : "forward tiles", pass == 0 ? tr : c, t, w);
  }
  if (!why.empty()) return fail(BBTC_ERR_LAYOUT, "device layout check failed: " + why);
  return BBTC_OK;
}
