// Intersection kernels, the device work queue and the launch paths.
//
// A task (i, j, k) contributes sum_{r in part i} sum_{b in ab[r]} |ac[r] ∩ bc[b]|
// (the reference's SparseKernel / DenseKernel, src/triangle_counting/
// gpu_sparse_kernel.cu:6-49 and gpu_dense_kernel.cu:3-47, one thread per row
// of ab).  Here the sum is taken one *pivot row* at a time: the pivot row
// becomes a membership structure in the warp's shared memory and the rows it
// meets are streamed against it.
//
// Per-task execution (plain form, explicit task lists):
//   v-centric (default): pivot = row b of bc (vertex v of part j); the rows
//     streamed are ac[u] for every u with b in ab[u] -- column b of ab, read
//     from the reversed tile (j, i).  With the degree order the ac rows are the
//     shorter side, so this probes sum d_k(u) ids where the reference's bitmap
//     form probes sum d_k(v).
//   u-centric (the reference's row order, BBTC_KERNEL_MERGE): pivot = ac[r],
//     the rows bc[b] for b in ab[r] are streamed against it.
//
// The whole task list at once runs as pivot lists instead (fused.cu).
//
// Membership structures: a bitmap of the column part, a sorted copy searched
// by bisection, or -- for pivot rows longer than the shared buffer -- bisection
// in global memory.
//
// Work units are runs of `unit_edges` consecutive entries of the rows tile.
// In the persistent form every warp of a grid sized to the SM count claims
// units from one atomic head over all tasks (cost-sorted, heaviest first); in
// the plain form each task is one launch whose warps stride over its units.
// Inside a unit the rows met by 32 entries are concatenated and walked 32
// consecutive ids at a time (see probe_entries).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <sstream>

#include "deliver.cuh"
#include "internal.h"
#include "search.cuh"

namespace bbtc {

namespace {

constexpr uint32_t FULL = 0xffffffffu;
// per warp after its bitmap: 33 segment starts, 32 bases and the staging state
constexpr uint32_t kSegWords = 96;
// per-warp bulk-staging state of the per-task kernels, after the bitmap:
// an mbarrier (8 bytes) at kBarOffset, its phase bit and a "staging off" flag
constexpr uint32_t kBarOffset = 92;
constexpr uint32_t kPhaseOffset = 94;
constexpr uint32_t kStageOffFlag = 95;
constexpr uint32_t kStageMin = 64;         // pivot rows this long or longer are staged by one bulk copy
constexpr uint32_t kWaitLimit = 1u << 20;  // try_wait polls before a staging copy is given up
// values of the warp's staging flag (state[kStageOffFlag])
constexpr uint32_t kStageOn = 0, kStageOff = 1, kStageDead = 2;

// ---- bulk copies into shared memory (cp.async.bulk + mbarrier) ------------

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void bar_init(uint64_t* bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(bar)) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// One lane: copy `bytes` (a multiple of 16; both addresses 16-byte aligned)
// from global to shared memory, completing on `bar`.
__device__ __forceinline__ void bulk_to_shared(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // earlier plain stores to dst come first
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes)
               : "memory");
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_addr(dst)),
               "l"(src), "r"(bytes), "r"(smem_addr(bar))
               : "memory");
}

// Wait for the phase with parity `parity` of `bar` to complete; false when
// it has not after `limit` polls.  Warp-uniform: true only when every lane
// saw the phase complete (each lane's own wait orders its later reads).
__device__ __forceinline__ bool bar_wait(uint64_t* bar, uint32_t parity, uint32_t limit) {
  bool done_all = false;
  for (uint32_t i = 0; i < limit; i++) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(done)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    if (done) {
      done_all = true;
      break;
    }
  }
  return __all_sync(FULL, done_all);
}

struct PivotView {
  const uint32_t* row;  // global pivot row
  uint32_t len;
  uint32_t base;  // bitmap bit 0 <-> id `base`
  uint32_t cap;   // a bit of the warp's last buffer word, which stays zero
  uint32_t first, last;
};

template <uint32_t KIND>
__device__ __forceinline__ uint32_t member(const uint32_t* bm, const PivotView& pv, uint32_t x) {
  if constexpr (KIND == kPivotBitmap) {
    // ids outside the pivot's span (below base they wrap high) land on the
    // always-zero last word: no branch
    const uint32_t y = min(x - pv.base, pv.cap);
    return (bm[y >> 5] >> (y & 31)) & 1u;
  } else if constexpr (KIND == kPivotList) {
    if (x < pv.first || x > pv.last) return 0;
    const uint32_t p = lower_bound_u32(bm, pv.len, x);
    return (p < pv.len && bm[p] == x) ? 1u : 0u;
  } else {
    if (x < pv.first || x > pv.last) return 0;
    const uint32_t p = lower_bound_u32(pv.row, pv.len, x);
    return (p < pv.len && pv.row[p] == x) ? 1u : 0u;
  }
}

// Segment of the probe ids met by entry q of the rows tile.
struct TileSegs {  // per task: the probe tile's row r = rows.col[q]
  const uint32_t* __restrict__ rcol;
  const uint32_t* __restrict__ rp;
  __device__ __forceinline__ void get(uint32_t q, uint32_t& start, uint32_t& len) const {
    const uint32_t r = rcol[q];
    start = rp[r];
    len = rp[r + 1] - start;
  }
};
// Probe the rows met by entries [e, ee) against the pivot structure; returns
// this lane's hit count.
//
// The rows met by a batch of 32 entries are concatenated and walked 32 ids at
// a time, lane l taking ids l, l + 32, l + 64, ..., so each warp load reads
// consecutive ids.  Every lane keeps a pointer to the row that owns its
// current id (found once per batch by bisection of the 33 row starts in
// shared memory) and moves it forward when its id passes the row's end --
// less than once per window on average -- so the owner costs one compare per
// id.  Four windows are loaded before any is tested.
template <uint32_t KIND, class Segs>
__device__ __forceinline__ uint32_t probe_entries(const Segs& segs, uint32_t e, uint32_t ee,
                                                  const uint32_t* __restrict__ prb_col, const uint32_t* bm,
                                                  uint32_t* sstart, uint32_t* sbase, const PivotView& pv,
                                                  uint32_t lane) {
  uint32_t hits = 0;
  for (uint32_t base = e; base < ee; base += 32) {
    const uint32_t q = base + lane;
    uint32_t start = 0, len = 0;
    if (q < ee) segs.get(q, start, len);
    uint32_t incl = len;
#pragma unroll
    for (uint32_t d = 1; d < 32; d <<= 1) {
      const uint32_t t = __shfl_up_sync(FULL, incl, d);
      if (lane >= d) incl += t;
    }
    const uint32_t total = __shfl_sync(FULL, incl, 31);
    if (total == 0) continue;
    const uint32_t excl = incl - len;
    sstart[lane] = excl;
    sbase[lane] = start - excl;  // modular: sbase + id is the id's position for ids of this row
    if (lane == 31) sstart[32] = total;
    __syncwarp();
    // owner of id = lane: the last row whose start is <= lane (empty rows share starts)
    uint32_t owner = 0;
#pragma unroll
    for (uint32_t step = 16; step > 0; step >>= 1)
      if (sstart[owner + step] <= lane) owner += step;
    uint32_t nb = sstart[owner + 1];
    uint32_t bs = sbase[owner];
    uint32_t gown = 0xffffffffu, gpos = 0;  // global kind: probe row and position of the last search
    for (uint32_t c = 0; c < total; c += 128) {
      uint32_t x[4];
      bool ok[4];
      uint32_t own[4];
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const uint32_t id = c + 32u * k + lane;
        ok[k] = id < total;
        x[k] = 0;
        if (ok[k]) {
          while (id >= nb) {
            owner++;
            nb = sstart[owner + 1];
            bs = sbase[owner];
          }
          x[k] = __ldg(prb_col + bs + id);
        }
        own[k] = owner;
      }
      if constexpr (KIND == kPivotGlobal) {
        // galloping search in the pivot row from this lane's last position
        // in the same probe row (ids of one row come in increasing order)
#pragma unroll
        for (int k = 0; k < 4; k++) {
          if (!ok[k]) continue;
          if (own[k] != gown) {
            gown = own[k];
            gpos = 0;
          }
          if (x[k] < pv.first || x[k] > pv.last) continue;
          gpos = gallop_lb(pv.row, pv.len, gpos, x[k]);
          hits += (gpos < pv.len && pv.row[gpos] == x[k]) ? 1u : 0u;
        }
      } else {
#pragma unroll
        for (int k = 0; k < 4; k++) hits += ok[k] ? member<KIND>(bm, pv, x[k]) : 0u;
      }
    }
    __syncwarp();
  }
  return hits;
}

// Build the pivot structure, probe entries [e, ee), restore the buffer to zero.
template <uint32_t KIND, class Segs>
__device__ __forceinline__ uint32_t pivot_pass(const uint32_t* __restrict__ prow, uint32_t pd, uint32_t base,
                                               uint32_t words, const Segs& segs, uint32_t e,
                                               uint32_t ee, const uint32_t* __restrict__ prb_col, uint32_t* bm,
                                               uint32_t* sstart, uint32_t* sbase, uint32_t lane) {
  if constexpr (KIND == kPivotBitmap) {
    for (uint32_t i = lane; i < pd; i += 32) {
      const uint32_t y = prow[i] - base;
      atomicOr(&bm[y >> 5], 1u << (y & 31));
    }
  } else if constexpr (KIND == kPivotList) {
    for (uint32_t i = lane; i < pd; i += 32) bm[i] = prow[i];
  }
  __syncwarp();
  PivotView pv;
  pv.row = prow;
  pv.len = pd;
  pv.base = base;
  pv.cap = words * 32;  // callers keep words < the buffer size, so word `words` is never set
  pv.first = prow[0];
  pv.last = prow[pd - 1];
  const uint32_t hits = probe_entries<KIND>(segs, e, ee, prb_col, bm, sstart, sbase, pv, lane);
  // the buffer is all-zero between pivots whatever kind used it last: the
  // persistent queue hands one warp bitmap and list work in any order
  __syncwarp();
  if constexpr (KIND == kPivotBitmap) {
    if (pd < words) {
      for (uint32_t i = lane; i < pd; i += 32) bm[(prow[i] - base) >> 5] = 0;
    } else {
      for (uint32_t i = lane; i < words; i += 32) bm[i] = 0;
    }
  } else if constexpr (KIND == kPivotList) {
    for (uint32_t i = lane; i < pd; i += 32) bm[i] = 0;
  }
  __syncwarp();
  return hits;
}

// One per-task work unit: entries [unit*K, min((unit+1)*K, nnz)) of the rows tile.
// Per-task pivot of the bitmap or list kind, staged in shared memory by one
// bulk copy (cp.async.bulk, the TMA engine; completion on the warp's
// mbarrier) of the 16-byte aligned span of the pivot row's column ids: the
// bitmap is then set, and cleared afterwards, from shared memory, and the
// list kind searches the staged span in place.  Returns false, having done
// nothing, when the row is short, the span does not fit the room left in the
// warp's buffer, or staging is off on this warp; the caller then loads the
// row itself (pivot_pass).  The column segment of a tile starts on a 16-byte
// boundary and the pool ends with a 16-byte tail, so the rounded span stays
// inside the allocation.
//
// A copy that has not landed after the wait limit voids the count (the
// error word; the host fails the call with BBTC_ERR_TIMEOUT).  The warp then
// waits once more, bounded, for the copy still in flight: if it lands, the
// staged span is cleared and the warp goes on without staging; if not, the
// warp may not touch its buffer again and stops (kStageDead), taking no more
// work.  `dbg` > 0 is the test hook of bbtc_debug_stage_timeout: no copy is
// issued, so the wait gives up after `dbg` polls with nothing in flight.
template <uint32_t KIND>
__device__ __forceinline__ bool staged_pass(const uint32_t* __restrict__ tile_col, uint32_t ps, uint32_t pd,
                                            uint32_t words, const TileSegs& segs, uint32_t e, uint32_t ee,
                                            const uint32_t* __restrict__ prb_col, uint32_t* bm, uint32_t bm_words,
                                            uint32_t* sstart, uint32_t* sbase, uint32_t lane, uint32_t* err,
                                            uint32_t dbg, unsigned long long& acc) {
  uint32_t* state = bm + bm_words;
  if (pd < kStageMin || state[kStageOffFlag] != kStageOn) return false;
  const uint32_t a0 = ps & ~3u, off = ps & 3u;
  const uint32_t span = ((ps + pd + 3u) & ~3u) - a0;  // words, a multiple of 4
  // bitmap kind: after the bitmap and its always-zero word; list kind: the list itself
  uint32_t* stage = KIND == kPivotList ? bm : bm + ((words + 1u + 3u) & ~3u);
  if (span > bm_words - (uint32_t)(stage - bm)) return false;
  uint64_t* bar = reinterpret_cast<uint64_t*>(state + kBarOffset);
  const uint32_t phase = state[kPhaseOffset];
  const uint32_t limit = dbg ? dbg : kWaitLimit;
  if (lane == 0 && !dbg) bulk_to_shared(stage, tile_col + a0, span * 4u, bar);
  const bool ok = bar_wait(bar, phase, limit);
  __syncwarp();
  if (!ok) {
    // the copy did not land in time: the count is void
    if (lane == 0) atomicOr(err, 1u);
    const bool landed = bar_wait(bar, phase, limit);  // drain the copy still in flight
    if (landed) {
      for (uint32_t i = lane; i < span; i += 32) stage[i] = 0;
      if (lane == 0) {
        state[kPhaseOffset] = phase ^ 1u;
        state[kStageOffFlag] = kStageOff;
      }
    } else if (lane == 0) {
      state[kStageOffFlag] = kStageDead;
    }
    __syncwarp();
    return true;
  }
  if (lane == 0) state[kPhaseOffset] = phase ^ 1u;
  const uint32_t* ids = stage + off;
  if constexpr (KIND == kPivotBitmap) {
    for (uint32_t i = lane; i < pd; i += 32) {
      const uint32_t y = ids[i];
      atomicOr(&bm[y >> 5], 1u << (y & 31));
    }
  }
  __syncwarp();
  PivotView pv;
  pv.row = tile_col + ps;
  pv.len = pd;
  pv.base = 0;
  pv.cap = words * 32;
  pv.first = ids[0];
  pv.last = ids[pd - 1];
  const uint32_t hits =
      probe_entries<KIND>(segs, e, ee, prb_col, KIND == kPivotList ? ids : bm, sstart, sbase, pv, lane);
  __syncwarp();
  // back to an all-zero buffer: the bitmap words the ids set, then the staged span
  if constexpr (KIND == kPivotBitmap) {
    if (pd < words) {
      for (uint32_t i = lane; i < pd; i += 32) bm[ids[i] >> 5] = 0;
    } else {
      for (uint32_t i = lane; i < words; i += 32) bm[i] = 0;
    }
    __syncwarp();
  }
  for (uint32_t i = lane; i < span; i += 32) stage[i] = 0;
  __syncwarp();
  acc += hits;
  return true;
}

// Set up a warp's staging state (kernel start, before any bulk copy).
__device__ __forceinline__ void staging_init(uint32_t* bm, uint32_t bm_words, uint32_t lane) {
  uint32_t* state = bm + bm_words;
  if (lane == 0) {
    bar_init(reinterpret_cast<uint64_t*>(state + kBarOffset));
    state[kPhaseOffset] = 0;
    state[kStageOffFlag] = kStageOn;
  }
  __syncwarp();
}

// True once a staging copy of this warp was given up while possibly still in
// flight: the warp stops working (its count is void already).
__device__ __forceinline__ bool staging_dead(const uint32_t* bm, uint32_t bm_words) {
  return bm[bm_words + kStageOffFlag] == kStageDead;
}

__device__ __noinline__ unsigned long long task_unit(const DevTask& tk, uint32_t unit, uint32_t* bm,
                                                     uint32_t* sstart, uint32_t* sbase, uint32_t lane,
                                                     uint32_t bm_words, uint32_t* err, uint32_t dbg) {
  const uint32_t* __restrict__ r_rp = tk.rows.rp;
  const uint32_t* __restrict__ p_rp = tk.pivot.rp;
  const uint32_t* __restrict__ p_col = tk.pivot.col;
  const TileSegs segs{tk.rows.col, tk.probe.rp};
  const uint32_t H = tk.rows.H;
  const uint64_t e0 = (uint64_t)unit * tk.unit_edges;
  const uint64_t e1w = e0 + tk.unit_edges;
  uint32_t e = (uint32_t)e0;
  const uint32_t e1 = e1w < tk.rows.nnz ? (uint32_t)e1w : tk.rows.nnz;
  uint32_t b = tk.rows.erow[e >> 5];  // units start at multiples of 32 entries
  unsigned long long acc = 0;
  while (e < e1) {
    const uint32_t ee = min(r_rp[b + 1], e1);
    const uint32_t ps = p_rp[b];
    const uint32_t pd = p_rp[b + 1] - ps;
    if (pd > 0) {
      const uint32_t* prow = p_col + ps;
      switch (tk.kind) {
        case kPivotBitmap:
          if (!staged_pass<kPivotBitmap>(p_col, ps, pd, tk.words, segs, e, ee, tk.probe.col, bm, bm_words, sstart,
                                         sbase, lane, err, dbg, acc))
            acc += pivot_pass<kPivotBitmap>(prow, pd, 0, tk.words, segs, e, ee, tk.probe.col, bm, sstart,
                                                   sbase, lane);
          break;
        case kPivotList:
          if (!staged_pass<kPivotList>(p_col, ps, pd, 0, segs, e, ee, tk.probe.col, bm, bm_words, sstart, sbase, lane,
                                       err, dbg, acc))
            acc += pivot_pass<kPivotList>(prow, pd, 0, 0, segs, e, ee, tk.probe.col, bm, sstart, sbase, lane);
          break;
        default:
          acc += pivot_pass<kPivotGlobal>(prow, pd, 0, 0, segs, e, ee, tk.probe.col, bm, sstart, sbase, lane);
      }
      if (staging_dead(bm, bm_words)) return acc;
    }
    e = ee;
    if (e < e1) b = next_row(r_rp, H, b, e, lane);
  }
  return acc;
}

__device__ __forceinline__ unsigned long long warp_sum(unsigned long long v) {
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(FULL, v, d);
  return v;
}

// Persistent form: every warp claims units from one head until the queue is
// empty.  MINB is the register budget's occupancy target (blocks per SM).
template <int MINB>
__global__ void __launch_bounds__(256, MINB) k_count_queue(const DevTask* __restrict__ tasks,
                                                        const uint32_t* __restrict__ prefix, uint32_t ntasks,
                                                        uint32_t total_units, unsigned long long* __restrict__ outs,
                                                        uint32_t nouts, uint64_t* __restrict__ dev,
                                                        uint64_t* __restrict__ host, uint32_t bm_words, uint32_t dbg) {
  extern __shared__ __align__(16) uint32_t sh[];
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint32_t* bm = sh + warp * (bm_words + kSegWords);
  uint32_t* sstart = bm + bm_words;
  uint32_t* sbase = sstart + 33;
  uint32_t* head = reinterpret_cast<uint32_t*>(outs + nouts);
  uint32_t* err = head + 1;  // set when a staging copy gave up
  for (uint32_t i = lane; i < bm_words; i += 32) bm[i] = 0;
  staging_init(bm, bm_words, lane);
  while (true) {
    uint32_t g = 0;
    if (lane == 0) g = atomicAdd(head, 1u);
    g = __shfl_sync(FULL, g, 0);
    if (g >= total_units) break;
    uint32_t lo = 0, hi = ntasks;  // last t with prefix[t] <= g
    while (hi - lo > 1) {
      const uint32_t mid = (lo + hi) >> 1;
      if (prefix[mid] <= g) lo = mid; else hi = mid;
    }
    const DevTask& tk = tasks[lo];
    const unsigned long long c =
        warp_sum(task_unit(tk, g - prefix[lo], bm, sstart, sbase, lane, bm_words, err, dbg));
    if (lane == 0 && c) atomicAdd(&outs[tk.slot], c);
    if (staging_dead(bm, bm_words)) break;
  }
  if (host) deliver(outs, nouts, dev, host);
}

// Plain form: one task per launch; warps stride over the task's units.
__global__ void __launch_bounds__(256, 4) k_count_task(const DevTask* __restrict__ task, uint32_t units,
                                                       unsigned long long* __restrict__ outs, uint32_t bm_words,
                                                       uint32_t* __restrict__ err, uint32_t dbg) {
  extern __shared__ __align__(16) uint32_t sh[];
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint32_t* bm = sh + warp * (bm_words + kSegWords);
  uint32_t* sstart = bm + bm_words;
  uint32_t* sbase = sstart + 33;
  for (uint32_t i = lane; i < bm_words; i += 32) bm[i] = 0;
  staging_init(bm, bm_words, lane);
  const DevTask& tk = *task;
  const uint32_t wpb = blockDim.x >> 5;
  unsigned long long acc = 0;
  for (uint32_t u = blockIdx.x * wpb + warp; u < units; u += gridDim.x * wpb) {
    acc += task_unit(tk, u, bm, sstart, sbase, lane, bm_words, err, dbg);
    if (staging_dead(bm, bm_words)) break;
  }
  acc = warp_sum(acc);
  if (lane == 0 && acc) atomicAdd(&outs[tk.slot], acc);
}

size_t smem_bytes(uint32_t bm_words, uint32_t warps) {
  return (size_t)warps * (bm_words + kSegWords) * sizeof(uint32_t);
}

}  // namespace

size_t smem_bytes_for(const bbtc_opts& o) {
  return smem_bytes(norm_bm_words(o.bitmap_words), norm_warps(o.warps_per_block));
}

int kernel_smem_optin(bbtc_ctx* ctx, const bbtc_opts& o) {
  const uint32_t bmw = norm_bm_words(o.bitmap_words), wpb = norm_warps(o.warps_per_block);
  const size_t sm = std::max(smem_bytes(bmw, wpb), pivots_smem(bmw, wpb));
  if (sm > ctx->smem_optin)
    return fail(BBTC_ERR_ARG, "bitmap_words x warps_per_block needs " + std::to_string(sm) +
                                  " bytes of shared memory; the device allows " + std::to_string(ctx->smem_optin));
  if (sm <= ctx->smem_set) return BBTC_OK;
  // A kernel has one limit per device, whichever context launches it: it is
  // only ever raised, so what a context found once holds.  The kernels' own
  // attribute is asked, which a reset of the device takes back; it is raised
  // for k_count_task last.
  static std::mutex mu;
  std::lock_guard<std::mutex> lk(mu);
  cudaFuncAttributes now;
  BBTC_CUDA(cudaFuncGetAttributes(&now, k_count_task));
  if ((size_t)now.maxDynamicSharedSizeBytes < sm) {
    BBTC_TRY(pivots_smem_optin(sm));
    BBTC_CUDA(cudaFuncSetAttribute(k_count_queue<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    BBTC_CUDA(cudaFuncSetAttribute(k_count_queue<6>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    BBTC_CUDA(cudaFuncSetAttribute(k_count_queue<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    BBTC_CUDA(cudaFuncSetAttribute(k_count_task, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
  }
  ctx->smem_set = sm;
  return BBTC_OK;
}

// Queue of a fused request: its graphs, the largest first.  A graph's units
// are first single batches of 32 entries, where the layout found short in-lists
// (a batch there holds many pivots and takes longest), then 8, 4, 2 and 1
// batches: a larger unit builds its pivot less often (R-MAT s20 1.03 ms with
// single batches throughout, 0.89 with fours), a smaller one evens out the
// queue's end, so each size is kept until about two units of it per warp are
// left.  o.unit_work asks for one size throughout.
static int make_pivot_plan(const bbtc_ctx* ctx, const std::vector<bbtc_graph*>& graphs, const bbtc_opts& o, Plan* plan) {
  uint64_t left = 0;  // batches from the current graph on
  for (const bbtc_graph* g : graphs) left += (g->m + 31) / 32;
  uint64_t entries = 0, pivots = 0;
  for (const bbtc_graph* g : graphs) {
    entries += g->m;
    pivots += g->npiv;
  }
  const uint64_t warps = (uint64_t)ctx->sms * 40;  // about as many as run at once
  std::vector<uint32_t> order(graphs.size());
  for (uint32_t q = 0; q < order.size(); q++) order[q] = q;
  std::stable_sort(order.begin(), order.end(), [&](uint32_t a, uint32_t b) { return graphs[a]->m > graphs[b]->m; });
  plan->tasks.clear();
  plan->pivots.clear();
  plan->prefix.assign(1, 0);
  uint64_t total = 0;
  for (uint32_t q : order) {
    const bbtc_graph* g = graphs[q];
    if (!g->m || !g->npiv) {
      left -= (g->m + 31) / 32;
      continue;
    }
    PivotGraph d{};
    d.words = reinterpret_cast<const uint2*>(g->d_words);
    d.rec = reinterpret_cast<const uint2*>(g->d_rec);
    d.piv = static_cast<const uint4*>(g->d_piv);
    d.crow = g->d_crow;
    d.entries = (uint32_t)g->m;
    d.npiv = g->npiv;
    d.plain = g->oriented ? 1 : 0;
    d.slot = q;
    const uint64_t batches = (g->m + 31) / 32;  // 64-bit: m may be near 2^32
    if (o.unit_work) {  // about half a row is streamed per entry
      const double avg = std::max(1.0, 0.5 * (double)g->m / std::max(1u, g->n));
      d.level_size[0] = (uint32_t)std::min(512.0, std::max(1.0, std::ceil(o.unit_work / avg / 32)));
      d.level_units[0] = (uint32_t)((batches + d.level_size[0] - 1) / d.level_size[0]);
      total += d.level_units[0];
    } else {
      const uint64_t sparse = std::min<uint64_t>(g->sparse_end, batches);
      d.level_size[0] = 1;
      d.level_units[0] = (uint32_t)sparse;
      total += sparse;
      uint64_t rest = batches - sparse, after = left - batches;
      for (int l = 1; l < kLevels; l++) {
        const uint64_t size = 1ull << (kLevels - 1 - l);  // 8, 4, 2, 1
        const uint64_t keep = 2 * warps * size;           // batches that smaller units are kept for
        uint64_t units = rest + after > keep ? std::min(rest, rest + after - keep) / size : 0;
        if (l == kLevels - 1) units = rest;
        d.level_size[l] = (uint32_t)size;
        d.level_units[l] = (uint32_t)units;
        total += units;
        rest -= units * size;
      }
    }
    left -= batches;
    // every warp claims one unit past the end: leave room in the 32-bit head
    if (total >= 0xffff0000ull) return fail(BBTC_ERR_UNSUPPORTED, "about 2^32 work units or more in one request");
    plan->pivots.push_back(d);
    plan->prefix.push_back((uint32_t)total);
  }
  plan->total_units = (uint32_t)total;
  plan->fused = true;
  // four rows in flight instead of two where pivots have 32 in-edges or more on
  // average: R-MAT s22 (88) 5.53 -> 4.97 ms; but Chung-Lu 2^20 (20) 478 -> 504
  // us, geometric 2^18 (6) 157 -> 194
  plan->long_lists = entries >= 32 * pivots;
  return BBTC_OK;
}

// Unit sizes of the per-task kernels.  Units of 8192 probes were a few
// thousand per request and left the chip to the last ones: half the task list
// of R-MAT s18 / s15 / Chung-Lu 2^18 (bitmap kernel, us) 821 / 482 / 5318;
// 1024 probes, and at least eight units a warp, 549 / 111 / 472; 512 probes
// 587 / 112 / 481.
constexpr uint32_t kUnitWork = 1024;  // probes of a unit
constexpr uint32_t kUnitShare = 8;    // units per warp at least, while they hold 32 entries or more

// Build the device task array for a per-task request.  A single graph keeps
// the caller's task order (its border split); several graphs are merged into
// one queue ordered by estimated probe work, heaviest first.
static int make_plan(const bbtc_ctx* ctx, const std::vector<bbtc_graph*>& graphs,
                     const std::vector<std::vector<bbtc_task>>& tasks, const bbtc_opts& o, Plan* plan) {
  const uint32_t bmw = norm_bm_words(o.bitmap_words);
  const uint32_t unit_work = o.unit_work ? o.unit_work : kUnitWork;
  std::vector<DevTask> list;
  std::vector<double> cost;
  auto add = [&](DevTask d, double avg_probe) {
    uint32_t K = (uint32_t)std::min(16384.0, std::max(32.0, unit_work / std::max(1.0, avg_probe)));
    K = (K + 31) & ~31u;
    d.unit_edges = K;
    list.push_back(d);
    cost.push_back((double)d.rows.nnz * std::max(1.0, avg_probe));
  };
  for (size_t gi = 0; gi < graphs.size(); gi++) {
    const bbtc_graph* g = graphs[gi];
    const uint32_t P = g->P;
    for (const bbtc_task& t : tasks[gi]) {
      if (t.ab >= P * P || t.bc >= P * P || t.ac >= P * P)
        return fail(BBTC_ERR_ARG, "task names a tile outside the P x P grid");
      const uint32_t i = t.ab / P, j = t.ab % P, k = t.bc % P;
      if (t.bc / P != j || t.ac != i * P + k)
        return fail(BBTC_ERR_ARG, "task tiles are not of the form (i,j), (j,k), (i,k)");
      if (!g->fwd.nnz[t.ab] || !g->fwd.nnz[t.bc] || !g->fwd.nnz[t.ac]) continue;  // bb_tc.cpp:86-91
      DevTask d{};
      const bool u_centric = (o.kernel == BBTC_KERNEL_MERGE);
      if (u_centric) {
        d.rows = dev_tile(g->fwd, g->cuts, i, j);
        d.pivot = dev_tile(g->fwd, g->cuts, i, k);
        d.probe = dev_tile(g->fwd, g->cuts, j, k);
      } else {
        d.rows = dev_tile(g->rev, g->cuts, j, i);
        d.pivot = dev_tile(g->fwd, g->cuts, j, k);
        d.probe = dev_tile(g->fwd, g->cuts, i, k);
      }
      d.words = (d.pivot.W + 31) / 32;
      const bool fits_bitmap = d.words < bmw;  // the word after the part stays zero
      const bool fits_list = d.pivot.maxdeg <= bmw;
      if (!u_centric && o.kernel != BBTC_KERNEL_SEARCH && fits_bitmap)
        d.kind = kPivotBitmap;
      else
        d.kind = fits_list ? kPivotList : kPivotGlobal;
      d.slot = (uint32_t)gi;
      const uint32_t probe_tile = u_centric ? j * P + k : i * P + k;
      const uint32_t probe_rows = std::max<uint32_t>(1, g->fwd.nerows[probe_tile]);
      add(d, (double)d.probe.nnz / probe_rows);
    }
  }
  if (!o.unit_work) {
    // no unit larger than an even share of the launch's entries -- the whole
    // queue's, or in the plain form the task's -- over a few units per warp
    const uint64_t warps = (uint64_t)ctx->sms * 32;
    uint64_t entries = 0;
    for (const DevTask& d : list) entries += d.rows.nnz;
    for (DevTask& d : list) {
      const uint64_t share = o.mode == BBTC_MODE_PLAIN ? d.rows.nnz / (2 * warps) : entries / (kUnitShare * warps);
      d.unit_edges = std::min(d.unit_edges, ((uint32_t)std::min<uint64_t>(share, 16384) + 31) & ~31u);
      d.unit_edges = std::max(d.unit_edges, 32u);
    }
  }
  std::vector<uint32_t> order(list.size());
  for (uint32_t q = 0; q < order.size(); q++) order[q] = q;
  if (graphs.size() > 1)
    std::stable_sort(order.begin(), order.end(), [&](uint32_t a, uint32_t b) { return cost[a] > cost[b]; });
  plan->tasks.clear();
  plan->pivots.clear();
  plan->prefix.assign(1, 0);
  uint64_t total = 0;
  for (uint32_t q : order) {
    const DevTask& d = list[q];
    total += ((uint64_t)d.rows.nnz + d.unit_edges - 1) / d.unit_edges;  // 64-bit: nnz may be near 2^32
    if (total >= 0xffffffffull) return fail(BBTC_ERR_UNSUPPORTED, "more than 2^32 work units in one request");
    plan->tasks.push_back(d);
    plan->prefix.push_back((uint32_t)total);
  }
  plan->total_units = (uint32_t)total;
  plan->fused = false;
  return BBTC_OK;
}

void Plan::release() {
  if (exec) cudaGraphExecDestroy(exec);
  if (d_queue) cudaFreeAsync(d_queue, stream);
  exec = nullptr;
  d_queue = nullptr;
  cap = 0;
}

static int enqueue_launches(bbtc_ctx* ctx, Plan* plan, const bbtc_opts& o, uint64_t* d_outs, uint32_t nouts,
                            const Delivery* to) {
  cudaStream_t s = ctx->stream;
  const uint32_t bmw = norm_bm_words(o.bitmap_words);
  const uint32_t wpb = norm_warps(o.warps_per_block);
  const size_t sm = smem_bytes(bmw, wpb);
  plan->launches = 0;
  const uint32_t ntasks = (uint32_t)plan->prefix.size() - 1;
  if ((!plan->fused && o.mode == BBTC_MODE_PLAIN) || ntasks == 0) to = nullptr;
  plan->delivers = to != nullptr;
  // the counts and, after them, the control word: queue head, staging flag
  if (!to) BBTC_CUDA(cudaMemsetAsync(d_outs, 0, (nouts + 1) * sizeof(uint64_t), s));
  uint64_t* acc = to ? to->acc : d_outs;
  uint64_t* dev = to ? to->dev : nullptr;
  uint64_t* host = to ? to->host : nullptr;
  if (ntasks == 0) return BBTC_OK;
  const uint32_t* d_prefix = reinterpret_cast<const uint32_t*>(static_cast<const char*>(plan->d_queue) + plan->prefix_at);
  if (plan->fused) {
    BBTC_TRY(pivots_launch(ctx, plan->pivots[0], static_cast<const PivotGraph*>(plan->d_queue), d_prefix, ntasks,
                           plan->total_units, plan->long_lists, o, acc, nouts, dev, host));
    plan->launches = 1;
    return BBTC_OK;
  }
  const DevTask* d_tasks = static_cast<const DevTask*>(plan->d_queue);
  if (o.mode == BBTC_MODE_PLAIN) {
    uint32_t* err = reinterpret_cast<uint32_t*>(d_outs + nouts) + 1;
    for (uint32_t t = 0; t < ntasks; t++) {
      const uint32_t units = plan->prefix[t + 1] - plan->prefix[t];
      const uint32_t grid = std::max<uint32_t>(1, std::min<uint32_t>((units + wpb - 1) / wpb, ctx->sms * 8));
      k_count_task<<<grid, wpb * 32, sm, s>>>(d_tasks + t, units, reinterpret_cast<unsigned long long*>(d_outs), bmw,
                                               err, ctx->debug_stage_polls);
      BBTC_CUDA(cudaGetLastError());
      plan->launches++;
    }
  } else {
    // the register budget: 4, 6 or 8 resident blocks per SM
    const uint32_t occ = o.occupancy >= 8 ? 8 : (o.occupancy >= 6 ? 6 : 4);
    auto* qkern = occ == 8 ? k_count_queue<8> : (occ == 6 ? k_count_queue<6> : k_count_queue<4>);
    int per_sm = 0;
    BBTC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, qkern, wpb * 32, sm));
    per_sm = std::max(1, per_sm);
    if (o.blocks_per_sm) per_sm = std::min<int>(per_sm, (int)o.blocks_per_sm);
    // no more blocks than the queue has units for a warp each (a small batch
    // leaves the rest of the GPU to other streams)
    const uint64_t want = ((uint64_t)plan->total_units + wpb - 1) / wpb;
    const uint32_t grid = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>((uint64_t)ctx->sms * per_sm, want));
    qkern<<<grid, wpb * 32, sm, s>>>(d_tasks, d_prefix, ntasks, plan->total_units,
                                     reinterpret_cast<unsigned long long*>(acc), nouts, dev, host, bmw,
                                     ctx->debug_stage_polls);
    BBTC_CUDA(cudaGetLastError());
    plan->launches = 1;
  }
  return BBTC_OK;
}

int control_status(uint64_t ctrl) {
  if (ctrl >> 32) return fail(BBTC_ERR_TIMEOUT, "a shared-memory staging copy did not complete; the count is void");
  return BBTC_OK;
}

// Options left at 0 ("auto") resolved.  The buffer: 1024 words per warp
// (wider pivots run as rank bitmaps or hashes, so a larger buffer only costs
// occupancy).  Occupancy: the fused count 5 blocks per SM while the buffer
// leaves shared memory for them (R-MAT s22 / s20 / Chung-Lu 2^23, ms: 4 blocks
// 6.19 / 0.95 / 4.99, 5 blocks 5.61 / 0.91 / 4.76, 6 blocks 5.88 / 0.88 /
// 4.94), else 4 (64 registers); per-task kernels 4 (R-MAT s20: bitmap 10.4 ms
// at 4 against 12.4 at 6, search 14.4 / 15.7, merge 27.5 / 31.5).
static bbtc_opts resolve_opts(const bbtc_opts& in, bool fused) {
  bbtc_opts o = in;
  if (!o.bitmap_words) o.bitmap_words = 1024;
  if (!o.occupancy) o.occupancy = fused && norm_bm_words(o.bitmap_words) <= 1024 ? 5 : 4;
  return o;
}

int count_enqueue(bbtc_ctx* ctx, const std::vector<bbtc_graph*>& graphs,
                  const std::vector<std::vector<bbtc_task>>& tasks, const bbtc_opts& in, bool fused,
                  uint64_t* d_outs, Plan* plan, bool reuse, const Delivery* to) {
  Range range("bbtc count enqueue");
  cudaStream_t s = ctx->stream;
  const bbtc_opts o = resolve_opts(in, fused);
  BBTC_TRY(kernel_smem_optin(ctx, o));
  if (!reuse) {
    if (plan->exec) cudaGraphExecDestroy(plan->exec);
    plan->exec = nullptr;
    if (fused) BBTC_TRY(make_pivot_plan(ctx, graphs, o, plan));
    else BBTC_TRY(make_plan(ctx, graphs, tasks, o, plan));
    // one graph's fused queue rides in the kernel's arguments; other queues are uploaded
    const size_t nt = fused && plan->pivots.size() == 1 ? 0 : plan->prefix.size() - 1;
    if (nt) {
      const void* items = fused ? static_cast<const void*>(plan->pivots.data()) : plan->tasks.data();
      const size_t tb = nt * (fused ? sizeof(PivotGraph) : sizeof(DevTask)), pb = (nt + 1) * sizeof(uint32_t);
      if (tb + pb > plan->cap || plan->stream != s) {
        plan->release();
        plan->stream = s;
        const size_t cap = std::max<size_t>(tb + pb, 64 << 10);
        if (dev_malloc(&plan->d_queue, cap, s) != cudaSuccess) {
          cudaGetLastError();
          plan->release();
          return fail(BBTC_ERR_NOMEM, "device allocation of the task queue failed");
        }
        plan->cap = cap;
      }
      plan->prefix_at = tb;
      // upload from the context's pinned staging (a pageable copy would go
      // through the driver's shared staging buffers, which other threads'
      // copies hold); the context keeps it across plans, since pinning host
      // memory can take milliseconds
      if (ctx->h_plan_done) BBTC_CUDA(cudaEventSynchronize(ctx->h_plan_done));  // the last upload has read it
      if (tb + pb > ctx->h_plan_cap) {
        if (ctx->h_plan) cudaFreeHost(ctx->h_plan);
        ctx->h_plan = nullptr;
        ctx->h_plan_cap = 0;
        const size_t want = std::max<size_t>(tb + pb, 64 << 10) * 2;
        BBTC_CUDA(cudaMallocHost(&ctx->h_plan, want));
        ctx->h_plan_cap = want;
      }
      if (!ctx->h_plan_done) BBTC_CUDA(cudaEventCreateWithFlags(&ctx->h_plan_done, cudaEventDisableTiming));
      std::memcpy(ctx->h_plan, items, tb);
      std::memcpy(ctx->h_plan + tb, plan->prefix.data(), pb);
      BBTC_CUDA(cudaMemcpyAsync(plan->d_queue, ctx->h_plan, tb + pb, cudaMemcpyHostToDevice, s));
      BBTC_CUDA(cudaEventRecord(ctx->h_plan_done, s));
    }
    plan->captured = false;
  }
  if (plan->stage_polls != ctx->debug_stage_polls && plan->exec) {  // the launches take it as an argument
    cudaGraphExecDestroy(plan->exec);
    plan->exec = nullptr;
    plan->captured = false;
  }
  plan->stage_polls = ctx->debug_stage_polls;
  // A plan of one launch is launched directly (a memset and a kernel cost
  // less host time than a graph launch), and so is any plan's first count:
  // capturing and instantiating a graph pays only on replays, so the capture
  // waits for the plan's second count.
  if (!o.use_cuda_graph || !reuse || plan->fused || o.mode != BBTC_MODE_PLAIN)
    return enqueue_launches(ctx, plan, o, d_outs, (uint32_t)graphs.size(), to);
  if (!plan->captured) {
    cudaGraph_t graph = nullptr;
    BBTC_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
    const int rc = enqueue_launches(ctx, plan, o, d_outs, (uint32_t)graphs.size(), nullptr);
    const cudaError_t ec = cudaStreamEndCapture(s, &graph);
    if (rc != BBTC_OK) {
      if (graph) cudaGraphDestroy(graph);
      return rc;
    }
    if (ec != cudaSuccess) return cuda_fail(ec, "cudaStreamEndCapture");
    const cudaError_t ei = cudaGraphInstantiate(&plan->exec, graph, 0);
    cudaGraphDestroy(graph);
    if (ei != cudaSuccess) return cuda_fail(ei, "cudaGraphInstantiate");
    plan->captured = true;
  }
  BBTC_CUDA(cudaGraphLaunch(plan->exec, s));
  return BBTC_OK;
}

}  // namespace bbtc
