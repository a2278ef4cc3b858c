// The fused count: every task of the list in one pass over pivot lists.
//
// The tasks (i, j, k) for all k >= j share tile ab = (i, j), and the sum over
// all tasks (the reference's SparseKernel / DenseKernel over its task list,
// src/triangle_counting/gpu_sparse_kernel.cu:6-49, gpu_dense_kernel.cu:3-47)
// is the sum over edges (u, v) with part(u) <= part(v) of
// |N+(u) ∩ N+(v) ∩ [cuts[part(v)], ∞)|.  The layout (layout.cu) lists, per
// pivot v, its in-edges (u, v) with the range of N+(u)'s (word, mask) pairs
// that can meet N+(v); a warp makes N+(v) a membership structure in its
// shared memory and streams those pairs against it.
//
// What bounds it: instruction issue and the L1 / shared-memory pipe (R-MAT s20:
// issue 72 %, that pipe 76 %, DRAM at 14 % of the copy rate): every streamed
// pair is one 8-byte global load and one random shared-memory read.  So the
// work around the pairs is what the design keeps small:
//   * no tiles: a pivot's in-edges lie together whatever the cut vector, and
//     only vertices that are pivots are listed, so no warp walks empty row
//     pointers (that had left the SMs idle for 30 % of the s20 count);
//   * lanes own rows (32, or 8 side by side when rows are short), so no lane
//     searches the row that its pair belongs to; the batch's rows are read from
//     shared memory, one 8-byte broadcast a row (shuffles took two);
//   * in-lists of a few entries share one hash table per run, so 32 entries
//     cost two rounds of loads and not two per pivot;
//   * units of up to eight batches of 32 entries where in-lists are long (the
//     pivot is rebuilt per unit), of one batch where they are short or the
//     queue ends;
//   * the state between the probe loops lives in shared memory, and what is one
//     call's is inlined: the loops fit 48 registers (5 blocks of 8 warps on an
//     SM) and few registers are saved around them.  Where the loops are
//     functions, the bitmap's, hash's and search's spill nothing, the rank's and
//     the run's 16 bytes a call, and the kernel around them 136; inlined, 28 in
//     all.
// Per count, against the tiled task rows that this replaced (B200, ms): R-MAT
// s22 7.09 -> 4.85, s20 1.86 -> 0.78, s16 0.160 -> 0.074, s12 0.095 -> 0.032,
// Chung-Lu 2^23 17.5 -> 3.68, geometric 2^18 0.432 -> 0.105 (result included).
#include <algorithm>
#include <cstring>

#include "deliver.cuh"
#include "internal.h"

namespace bbtc {
namespace {

constexpr uint32_t FULL = 0xffffffffu;

// Membership structures of a pivot, chosen per pivot by its span and length.
// A pivot with this many entries in a batch of 32 gets a structure of its own;
// consecutive shorter ones share a hash table (run).  Where in-lists are short
// (8 / 12 / 16 / 24, ms: Chung-Lu 2^23 4.42 / 4.30 / 4.27 / 4.27, geometric
// 2^18 0.143 / 0.125 / 0.120 / 0.119) building costs more than probing; where
// they are long (R-MAT s22 4.96 / 5.00 / 5.02 / 5.03) the own structure, mostly
// a bitmap, is cheaper to probe.
constexpr uint32_t kAlone = 16, kAloneLong = 8;
constexpr uint32_t kRunSlots = 4;  // hash slots per pair of a run: chains stay short (2 measured 1-2 % slower)

enum PivotKind : uint32_t {
  kNone = 0,   // not built
  kBitmap,     // one bit per id of the row's word-aligned span
  kRank,       // per 32 words of span a (presence bits, first pair) entry, then the masks in pair order
  kHash,       // open-addressing table of (word + 1, mask) entries
  kSearch,     // too long for the buffer: bisection of the row's pairs in global memory
};

// Per-warp state in shared memory, so that the probe loops keep the register
// budget: one lane writes, every lane reads after a __syncwarp.
struct Frame {
  uint32_t p0, p1, ws, wn;     // the pivot: its entries, its row's pairs,
  uint32_t fw, span, mask0, v; // first word, words up to the last one, bits kept of the first pair, vertex
  const uint2* words;
  const uint2* rec;
  const uint4* piv;
  uint32_t k, slot, e1;
  uint32_t kind;
  uint32_t cap;  // rank: blocks of 32 words; hash: slots - 1
  uint32_t far;  // hash: longest displacement of an entry
  uint32_t npiv, plain;
  uint32_t pad[2];
  uint2 entry[32];  // the batch's entries: first pair and number of pairs of each one's row
};
constexpr uint32_t kFrameWords = sizeof(Frame) / 4;

// A warp's shared memory, named by its first word: its frame, then the buffer
// of the pivot's structure.  Functions that are not inlined take that index
// and address the array itself, so that their accesses stay shared-memory ones.
extern __shared__ __align__(16) uint32_t sh_mem[];
__device__ __forceinline__ Frame* frame(uint32_t at) { return reinterpret_cast<Frame*>(sh_mem + at); }
__device__ __forceinline__ uint32_t* buffer(uint32_t at) { return sh_mem + at + kFrameWords; }
static_assert(sizeof(Frame) % 16 == 0, "the bitmaps stay 16-byte aligned");

struct View {  // what a probe of one kind reads of the frame
  uint32_t fw, span, cap, far;
};

template <uint32_t KIND>
__device__ __forceinline__ uint32_t hits_of(const uint32_t* bm, const View& pv, const Frame* fr, uint2 w) {
  if constexpr (KIND == kBitmap) {
    // words outside the span (below the first they wrap high) land on word `span`, which stays zero
    return __popc(w.y & bm[min(w.x - pv.fw, pv.span)]);
  } else if constexpr (KIND == kRank) {
    const uint32_t rel = w.x - pv.fw;  // words below the first wrap high
    if (rel >= pv.span) return 0;
    const uint2 e = reinterpret_cast<const uint2*>(bm)[rel >> 5];
    const uint32_t bit = 1u << (rel & 31);
    if (!(e.x & bit)) return 0;
    return __popc(w.y & bm[2 * pv.cap + e.y + __popc(e.x & (bit - 1u))]);
  } else if constexpr (KIND == kHash) {
    const uint2* tab = reinterpret_cast<const uint2*>(bm);
    const uint32_t tag = w.x + 1u;
    for (uint32_t d = 0; d <= pv.far; d++) {
      const uint2 e = tab[(w.x + d) & pv.cap];
      if (e.x == tag) return __popc(w.y & e.y);
      if (e.x == 0) return 0;
    }
    return 0;
  } else {
    const uint2* __restrict__ row = fr->words + fr->ws;
    const uint32_t wn = fr->wn;
    uint32_t lo = 0, n = wn;  // first pair with word >= w.x
    while (n > 0) {
      const uint32_t half = n >> 1;
      if (row[lo + half].x < w.x) {
        lo += half + 1;
        n -= half + 1;
      } else {
        n = half;
      }
    }
    if (lo >= wn) return 0;
    const uint2 p = row[lo];
    return p.x == w.x ? __popc(w.y & (lo == 0 ? p.y & fr->mask0 : p.y)) : 0u;
  }
}

// Rows of the batch's entries [a, b), G lanes to a row, R rows of each lane
// group and two steps of each in flight.  R is 4 where the loads in flight
// decide (LONG: graphs of long in-lists, bitmap and rank pivots), else 2: the
// registers that 4 rows take are missing in the runs of short in-lists.
template <uint32_t KIND, bool LONG, uint32_t G>
__device__ __forceinline__ uint32_t probe_rows(uint32_t at, uint32_t a, uint32_t b) {
  constexpr uint32_t E = 32 / G;  // rows side by side
  constexpr uint32_t R = LONG && (KIND == kBitmap || KIND == kRank) ? 4 : 2, S = 2;
  const uint32_t lane = threadIdx.x & 31;
  const Frame* fr = frame(at);
  const uint32_t* bm = buffer(at);
  const uint2* __restrict__ words = fr->words;
  const View pv{fr->fw, fr->span, fr->cap, fr->far};
  uint32_t hits = 0;
  for (uint32_t r = a + lane / G; r < b; r += R * E) {
    uint2 e[R];
    uint32_t lm = 0;
#pragma unroll
    for (uint32_t q = 0; q < R; q++) {
      e[q] = make_uint2(0, 0);
      if (q == 0 || r + q * E < b) e[q] = fr->entry[r + q * E];
      lm = max(lm, e[q].y);
    }
    for (uint32_t i = lane & (G - 1); i < lm; i += S * G) {
      uint2 x[R][S];
#pragma unroll
      for (uint32_t s = 0; s < S; s++)
#pragma unroll
        for (uint32_t q = 0; q < R; q++) {
          x[q][s] = make_uint2(0, 0);
          if (i + s * G < e[q].y) x[q][s] = __ldg(words + e[q].x + s * G + i);
        }
#pragma unroll
      for (uint32_t q = 0; q < R; q++) hits += hits_of<KIND>(bm, pv, fr, x[q][0]);
#pragma unroll
      for (uint32_t s = 1; s < S; s++)
        if (i + s * G < lm) {
#pragma unroll
          for (uint32_t q = 0; q < R; q++) hits += hits_of<KIND>(bm, pv, fr, x[q][s]);
        }
    }
  }
  return hits;
}

// Pairs per row from which a row gets all 32 lanes (28, 36, 40 and 44 measure
// within 1 %, 20 and 14 are 2 and 4 % slower at R-MAT s20).
constexpr uint32_t kWholeWarp = 40;

template <uint32_t KIND, bool LONG>
__device__ __forceinline__ uint32_t probe_here(uint32_t at, uint32_t a, uint32_t b) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t total = __reduce_add_sync(FULL, lane >= a && lane < b ? frame(at)->entry[lane].y : 0u);
  if (total == 0) return 0;
  if (total >= kWholeWarp * (b - a)) return probe_rows<KIND, LONG, 32>(at, a, b);
  return probe_rows<KIND, LONG, 8>(at, a, b);
}

// Where in-lists are long the four loops are functions, each with the whole
// register budget for its rows in flight; a pivot is probed over many entries
// per call.  Where they are short a call's saved registers cost more than the
// loops' spills (Chung-Lu 2^23: 3.97 ms as functions, 3.72 inlined; R-MAT s22:
// 4.84 and 5.20).
template <uint32_t KIND, bool LONG>
__device__ __noinline__ uint32_t probe_call(uint32_t at, uint32_t a, uint32_t b) {
  return probe_here<KIND, LONG>(at, a, b);
}

template <uint32_t KIND, bool LONG>
__device__ __forceinline__ uint32_t probe(uint32_t at, uint32_t a, uint32_t b) {
  if constexpr (LONG) return probe_call<KIND, LONG>(at, a, b);
  else return probe_here<KIND, LONG>(at, a, b);
}

template <bool LONG>
__device__ __forceinline__ uint32_t probe_kind(uint32_t at, uint32_t a, uint32_t b) {
  switch (frame(at)->kind) {
    case kBitmap: return probe<kBitmap, LONG>(at, a, b);
    case kRank: return probe<kRank, LONG>(at, a, b);
    case kHash: return probe<kHash, LONG>(at, a, b);
    default: return probe<kSearch, LONG>(at, a, b);
  }
}

// A run of short in-lists at once: the pivots of lanes [j, j2) (lane l holds
// the l-th pivot of the batch: its row's first pair ws, pairs wn, and the
// pairs `excl` of the run's pivots before it) share one hash table keyed by
// (word, pivot), so the run costs one round of loads for the table and one
// for the streamed rows, whatever the number of pivots.  Lane l also holds
// entry l of the batch; `pl` is its pivot, as a lane.  Words come in clusters
// (the graph's hubs), alike for all pivots: a multiplicative hash spreads them.
__device__ __forceinline__ uint32_t run_slot(uint32_t tag, uint32_t shift) { return (tag * 0x9E3779B1u) >> shift; }

__device__ __forceinline__ uint32_t run_hits(const uint2* tab, uint32_t shift, uint32_t far, uint2 w, uint32_t pl) {
  const uint32_t tag = ((w.x << 5) | pl) + 1u, cap = FULL >> shift;
  const uint32_t s = run_slot(tag, shift);
  for (uint32_t d = 0; d <= far; d++) {
    const uint2 e = tab[(s + d) & cap];
    if (e.x == tag) return __popc(w.y & e.y);
    if (e.x == 0) return 0;
  }
  return 0;
}

// Always 8 lanes a row: a second path of 32 lanes cost every run 2 to 3 %
// (Chung-Lu 2^23 4.25 -> 4.17 ms without it, geometric 2^18 0.119 -> 0.115),
// and so do paths of 4 or 16, or 4 rows in flight.
__device__ __forceinline__ uint32_t run_rows(const Frame* fr, const uint2* tab, uint32_t shift, uint32_t far,
                                             uint32_t pl, uint32_t a, uint32_t b) {
  const uint2* __restrict__ words = fr->words;
  constexpr uint32_t G = 8, E = 32 / G;
  const uint32_t lane = threadIdx.x & 31;
  uint32_t hits = 0;
  for (uint32_t r = a + lane / G; r < b + lane / G; r += 2 * E) {
    const uint32_t sub = lane & (G - 1);
    const uint32_t q0 = __shfl_sync(FULL, pl, r), q1 = __shfl_sync(FULL, pl, r + E);
    uint2 e0 = make_uint2(0, 0), e1 = e0;
    if (r < b) e0 = fr->entry[r];
    if (r + E < b) e1 = fr->entry[r + E];
    const uint2* __restrict__ p0 = words + (e0.x + sub);
    const uint2* __restrict__ p1 = words + (e1.x + sub);
    int32_t c0 = (int32_t)(e0.y - sub), c1 = (int32_t)(e1.y - sub);
    while (max(c0, c1) > 0) {
      uint2 x0, x1;
      if (c0 > 0) x0 = __ldg(p0);
      if (c1 > 0) x1 = __ldg(p1);
      if (c0 > 0) hits += run_hits(tab, shift, far, x0, q0);
      if (c1 > 0) hits += run_hits(tab, shift, far, x1, q1);
      c0 -= G;
      c1 -= G;
      p0 += G;
      p1 += G;
    }
  }
  return hits;
}

__device__ __forceinline__ uint32_t run_here(uint32_t at, uint32_t pl, uint32_t ws, uint32_t excl, uint32_t total,
                                             uint32_t j, uint32_t j2, uint32_t a, uint32_t b) {
  const uint32_t lane = threadIdx.x & 31;
  const uint2* __restrict__ words = frame(at)->words;
  const uint32_t shift = __clz(max(64u, kRunSlots * total) - 1);  // slots: a power of two, at least kRunSlots a pair
  const uint32_t cap = FULL >> shift;
  uint2* tab = reinterpret_cast<uint2*>(buffer(at));
  uint32_t far = 0;
  for (uint32_t c = 0; c < total; c += 32) {
    const uint32_t i = c + lane;
    uint32_t o = j;  // the pivot that owns pair i: the last with excl <= i
#pragma unroll
    for (uint32_t step = 16; step > 0; step >>= 1) {
      const uint32_t x = __shfl_sync(FULL, excl, o + step);
      if (o + step < j2 && x <= i) o += step;
    }
    const uint32_t from = __shfl_sync(FULL, ws, o) + i - __shfl_sync(FULL, excl, o);
    if (i < total) {
      const uint2 w = __ldg(words + from);
      const uint32_t tag = ((w.x << 5) | o) + 1u;
      uint32_t s = run_slot(tag, shift), d = 0;
      while (atomicCAS(&tab[s & cap].x, 0u, tag) != 0u) {
        s++;
        d++;
      }
      tab[s & cap].y = w.y;
      far = max(far, d);
    }
  }
  far = __reduce_max_sync(FULL, far);
  __syncwarp();
  const uint32_t hits = run_rows(frame(at), tab, shift, far, pl, a, b);
  __syncwarp();
  uint4* q = reinterpret_cast<uint4*>(tab);
  for (uint32_t i = lane; 2 * i <= cap; i += 32) q[i] = make_uint4(0, 0, 0, 0);
  __syncwarp();
  return hits;
}

// A function or not, as probe (batch of 96: 0.294 ms as a function, 0.285
// inlined; R-MAT s20: 0.78 and 0.80).
__device__ __noinline__ uint32_t run_call(uint32_t at, uint32_t pl, uint32_t ws, uint32_t excl, uint32_t total,
                                          uint32_t j, uint32_t j2, uint32_t a, uint32_t b) {
  return run_here(at, pl, ws, excl, total, j, j2, a, b);
}

template <bool LONG>
__device__ __forceinline__ uint32_t run(uint32_t at, uint32_t pl, uint32_t ws, uint32_t excl, uint32_t total,
                                        uint32_t j, uint32_t j2, uint32_t a, uint32_t b) {
  if constexpr (LONG) return run_call(at, pl, ws, excl, total, j, j2, a, b);
  else return run_here(at, pl, ws, excl, total, j, j2, a, b);
}

// Slots of a hash of wn entries: a power of two, at least four slots an entry.
__device__ __forceinline__ uint32_t hash_slots(uint32_t wn) { return max(32u, 1u << (32 - __clz(4 * wn - 1))); }

// Build the frame's pivot in the warp's all-zero buffer.
__device__ __forceinline__ void build(uint32_t at, uint32_t bm_words) {
  const uint32_t lane = threadIdx.x & 31;
  Frame* fr = frame(at);
  uint32_t* bm = buffer(at);
  const uint32_t wn = fr->wn, fw = fr->fw, span = fr->span, mask0 = fr->mask0;
  const uint2* __restrict__ row = fr->words + fr->ws;
  uint32_t kind = kSearch, cap = 0, far = 0;
  const uint32_t blocks = (span + 31) >> 5;
  if (span < bm_words) {
    kind = kBitmap;
    for (uint32_t i = lane; i < wn; i += 32) {
      const uint2 w = __ldg(row + i);
      bm[w.x - fw] = i == 0 ? (w.y & mask0) : w.y;
    }
  } else if (2 * blocks + wn <= bm_words) {
    kind = kRank;
    cap = blocks;
    for (uint32_t c = 0; c < wn; c += 32) {  // every lane runs every round: the shuffle needs them all
      const uint32_t i = c + lane;
      const uint2 w = i < wn ? __ldg(row + i) : make_uint2(fw, 0u);
      uint32_t prev = __shfl_up_sync(FULL, w.x, 1);
      if (lane == 0 && c > 0) prev = __ldg(row + c - 1).x;
      if (i < wn) {
        const uint32_t rel = w.x - fw, blk = rel >> 5;
        atomicOr(&bm[2 * blk], 1u << (rel & 31));
        if (i == 0 || ((prev - fw) >> 5) != blk) bm[2 * blk + 1] = i;
        bm[2 * blocks + i] = i == 0 ? (w.y & mask0) : w.y;
      }
    }
  } else if (wn <= bm_words && 2 * hash_slots(wn) <= bm_words) {
    kind = kHash;
    cap = hash_slots(wn) - 1;
    for (uint32_t i = lane; i < wn; i += 32) {
      const uint2 w = __ldg(row + i);
      uint32_t s = w.x & cap, d = 0;
      while (atomicCAS(&bm[2 * s], 0u, w.x + 1u) != 0u) {
        s = (s + 1) & cap;
        d++;
      }
      bm[2 * s + 1] = i == 0 ? (w.y & mask0) : w.y;
      far = max(far, d);
    }
    far = __reduce_max_sync(FULL, far);
  }
  if (lane == 0) {
    fr->kind = kind;
    fr->cap = cap;
    fr->far = far;
  }
  __syncwarp();
}

// Back to an all-zero buffer, and the frame to no pivot.
__device__ __forceinline__ void clear(uint32_t at) {
  __syncwarp();
  const uint32_t lane = threadIdx.x & 31;
  Frame* fr = frame(at);
  uint32_t* bm = buffer(at);
  uint32_t n = 0;  // words to clear as a range, from the buffer's start
  const uint32_t kind = fr->kind;
  if (kind == kBitmap) n = fr->span;
  else if (kind == kHash) n = 2 * (fr->cap + 1);
  else if (kind == kRank) n = 2 * fr->cap + fr->wn;
  uint4* q = reinterpret_cast<uint4*>(bm);
  for (uint32_t i = lane; 4 * i < n; i += 32) q[i] = make_uint4(0, 0, 0, 0);
  __syncwarp();
  if (lane == 0) fr->kind = kNone;
  __syncwarp();
}

// Start fetching a row of pairs [r.x, r.y) into L2: its first and its last
// line.  Chung-Lu 2^23 4.62 -> 4.40 ms (first line only: 4.52; the rows of a
// batch that other warps reach later: no more than its own).
__device__ __forceinline__ void touch_row(const uint2* words, uint2 r) {
  if (r.y <= r.x) return;
  asm volatile("prefetch.global.L2 [%0];" ::"l"(words + r.x));
  if (((r.y - 1) ^ r.x) & ~15u) asm volatile("prefetch.global.L2 [%0];" ::"l"(words + (r.y - 1)));
}

// The frame's next pivot: two lanes copy its 32 bytes.
__device__ __forceinline__ void load_pivot(uint32_t at, uint32_t k, uint32_t lane) {
  Frame* fr = frame(at);
  if (lane < 2) reinterpret_cast<uint4*>(&fr->p0)[lane] = __ldg(fr->piv + 2 * (uint64_t)k + lane);
  if (lane == 0) fr->k = k;
  __syncwarp();
}

// A batch [base, be) that is not wholly the built pivot's: its pivots, one a
// lane; one that goes on past the batch stays built (it is the batch's last).
// Returns this lane's hits.
template <bool LONG>
__device__ __forceinline__ uint32_t mixed(uint32_t at, uint32_t bm_words, uint32_t base, uint32_t be) {
  const uint32_t lane = threadIdx.x & 31;
  Frame* fr = frame(at);
  const uint32_t room = (1u << (31 - __clz(bm_words))) / (2 * kRunSlots);  // pairs of a run
  uint32_t hits = 0, np;
  bool more = false;
  do {
    const uint32_t k = fr->k;
    uint4 d = make_uint4(~0u, 0, 0, 0);
    if (k + lane < fr->npiv) d = __ldg(fr->piv + 2 * (uint64_t)(k + lane));
    np = __popc(__ballot_sync(FULL, d.x < be));
    const uint32_t a = min(max(d.x, base) - base, 32u), b = min(max(d.y, base) - base, be - base);
    const bool alone = d.x >= be || b <= a || b - a >= (LONG ? kAloneLong : kAlone) || d.y > be || d.w > room ||
                       !fr->plain || lane == 31 || (lane == 0 && fr->kind != kNone);
    const uint32_t single = __ballot_sync(FULL, alone);
    uint32_t cum = alone ? 0u : d.w;
#pragma unroll
    for (uint32_t s = 1; s < 32; s <<= 1) {
      const uint32_t x = __shfl_up_sync(FULL, cum, s);
      if (lane >= s) cum += x;
    }
    const uint32_t ws = d.z, ab = a << 8 | b;  // all that a lane keeps, with its scan, across the calls below
    for (uint32_t j = 0; j < np;) {
      if ((single >> j) & 1u) {
        const uint32_t abj = __shfl_sync(FULL, ab, j), aj = abj >> 8, bj = abj & 0xffu;
        if (fr->kind == kNone) {
          load_pivot(at, k + j, lane);
          build(at, bm_words);
        }
        if (bj > aj) hits += probe_kind<LONG>(at, aj, bj);
        more = fr->p1 > be;
        if (!more) clear(at);
        j++;
      } else {
        uint32_t excl = __shfl_up_sync(FULL, cum, 1);  // the scan, exclusive
        if (lane == 0) excl = 0;
        const uint32_t before = __shfl_sync(FULL, excl, j);
        // the run ends before the first later pivot that stands alone or does not fit
        const uint32_t stop = __ballot_sync(FULL, lane > j && (((single >> lane) & 1u) || cum - before > room));
        const uint32_t j2 = stop ? (uint32_t)__ffs(stop) - 1 : np;
        const uint32_t starts = __reduce_or_sync(FULL, lane >= j && lane < j2 ? 1u << (ab >> 8) : 0u);
        const uint32_t pl = j + __popc(starts & (FULL >> (31 - lane))) - 1;  // this entry's pivot
        // entries between the run's pivots belong to vertices without a row
        const uint32_t own_end = __shfl_sync(FULL, ab, pl) & 0xffu, run_start = __shfl_sync(FULL, ab, j) >> 8,
                       run_end = __shfl_sync(FULL, ab, j2 - 1) & 0xffu;
        if (lane >= own_end && lane > run_start && lane < run_end) fr->entry[lane].y = 0;
        __syncwarp();
        const uint32_t total = __shfl_sync(FULL, cum, j2 - 1) - before;
        hits += run<LONG>(at, pl, ws, excl - before, total, j, j2, run_start, run_end);
        j = j2;
      }
    }
    if (more) np--;
    __syncwarp();
    if (lane == 0) fr->k = k + np;
    __syncwarp();
    if (more) break;
  } while (np == 32);
  return hits;
}

template <int MINB, bool LONG>
__global__ void __launch_bounds__(256, MINB)
    k_count_pivots(const __grid_constant__ PivotGraph one, const PivotGraph* __restrict__ many,
                   const uint32_t* __restrict__ prefix, uint32_t ng, uint32_t total_units,
                   unsigned long long* __restrict__ outs, uint32_t nouts, uint64_t* __restrict__ dev,
                   uint64_t* __restrict__ host, uint32_t bm_words) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t at = (threadIdx.x >> 5) * (bm_words + kFrameWords);
  Frame* fr = frame(at);
  for (uint32_t i = lane; i < bm_words; i += 32) buffer(at)[i] = 0;
  uint32_t* head = reinterpret_cast<uint32_t*>(outs + nouts);
  uint32_t g = 0;
  if (lane == 0) g = atomicAdd(head, 1u);
  while (true) {
    g = __shfl_sync(FULL, g, 0);
    if (g >= total_units) break;
    const PivotGraph* gr = &one;
    uint32_t unit = g;
    if (ng > 1) {
      uint32_t lo = 0, hi = ng;  // last t with prefix[t] <= g
      while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (prefix[mid] <= g) lo = mid; else hi = mid;
      }
      gr = many + lo;
      unit -= prefix[lo];
    }
    // the unit's batches [q0, q1)
    uint32_t q0 = 0, size = 1, u = unit;
#pragma unroll
    for (int l = 0; l < kLevels; l++) {
      const uint32_t c = gr->level_units[l];
      size = gr->level_size[l];
      if (u < c || l == kLevels - 1) break;
      u -= c;
      q0 += c * size;
    }
    q0 += u * size;
    uint32_t base = q0 * 32;  // < entries < 2^32
    if (lane == 0) {
      fr->words = gr->words;
      fr->rec = gr->rec;
      fr->piv = gr->piv;
      fr->npiv = gr->npiv;
      fr->plain = gr->plain;
      fr->slot = gr->slot;
      fr->e1 = (gr->entries - base) / 32 >= size ? base + 32 * size : gr->entries;
      fr->kind = kNone;
      fr->k = __ldg(gr->crow + q0);
    }
    __syncwarp();
    unsigned long long acc = 0;
    while (true) {
      const uint32_t e1 = fr->e1;
      const uint32_t be = e1 - base > 32 ? base + 32 : e1;
      uint2 r = make_uint2(0, 0);
      if (base + lane < be) r = __ldg(fr->rec + base + lane);
      if (!LONG) touch_row(fr->words, r);  // while the pivots are read and their table is built
      fr->entry[lane] = make_uint2(r.x, r.y - r.x);
      __syncwarp();
      if (fr->kind != kNone && fr->p1 > be)
        acc += probe_kind<LONG>(at, 0, be - base);
      else
        acc += mixed<LONG>(at, bm_words, base, be);
      if (be == e1) break;
      base = be;
      __syncwarp();
    }
    if (fr->kind != kNone) clear(at);
    const uint32_t slot = fr->slot;
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) acc += __shfl_xor_sync(FULL, acc, d);
    if (lane == 0) {
      if (acc) atomicAdd(&outs[slot], acc);
      g = atomicAdd(head, 1u);
    }
    __syncwarp();
  }
  if (host) deliver(outs, nouts, dev, host);
}

using Kernel = void (*)(const PivotGraph, const PivotGraph*, const uint32_t*, uint32_t, uint32_t, unsigned long long*,
                        uint32_t, uint64_t*, uint64_t*, uint32_t);

Kernel kernel_for(uint32_t occ, bool long_lists) {
  if (occ >= 8) return k_count_pivots<8, false>;
  if (occ >= 6) return k_count_pivots<6, false>;
  if (occ == 5) return long_lists ? k_count_pivots<5, true> : k_count_pivots<5, false>;
  return k_count_pivots<4, false>;
}

}  // namespace

size_t pivots_smem(uint32_t bm_words, uint32_t warps) {
  return (size_t)warps * (bm_words + kFrameWords) * sizeof(uint32_t);
}

int pivots_smem_optin(size_t bytes) {
  for (Kernel k : {k_count_pivots<4, false>, k_count_pivots<5, false>, k_count_pivots<5, true>, k_count_pivots<6, false>,
                   k_count_pivots<8, false>})
    BBTC_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
  return BBTC_OK;
}

int pivots_launch(bbtc_ctx* ctx, const PivotGraph& one, const PivotGraph* d_many, const uint32_t* d_prefix, uint32_t ng,
                  uint32_t total_units, bool long_lists, const bbtc_opts& o, uint64_t* d_outs, uint32_t nouts,
                  uint64_t* dev, uint64_t* host) {
  const uint32_t bmw = norm_bm_words(o.bitmap_words), wpb = norm_warps(o.warps_per_block);
  const size_t sm = pivots_smem(bmw, wpb);
  const Kernel kern = kernel_for(o.occupancy, long_lists);
  int per_sm = 0;
  BBTC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, wpb * 32, sm));
  per_sm = std::max(1, per_sm);
  if (o.blocks_per_sm) per_sm = std::min<int>(per_sm, (int)o.blocks_per_sm);
  // no more blocks than the queue has units for a warp each (a small batch
  // leaves the rest of the GPU to other streams)
  const uint64_t want = ((uint64_t)total_units + wpb - 1) / wpb;
  const uint32_t grid = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>((uint64_t)ctx->sms * per_sm, want));
  kern<<<grid, wpb * 32, sm, ctx->stream>>>(one, d_many, d_prefix, ng, total_units,
                                            reinterpret_cast<unsigned long long*>(d_outs), nouts, dev, host, bmw);
  BBTC_CUDA(cudaGetLastError());
  return BBTC_OK;
}

}  // namespace bbtc
