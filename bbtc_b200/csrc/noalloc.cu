// Counting without allocation.
//
// bbtc_count_csr_noalloc counts the triangles of an oriented CSR that the
// caller already holds in device memory, for callers that cannot allocate
// device memory themselves or through this library: code that runs inside
// another framework's device-memory manager (which owns the device's memory
// and hands out only slices of its own pool), processes held to a fixed
// device-memory quota, and paths that must not pay cudaMalloc / cudaFree's
// implicit device synchronisation.  The CSR is one task in the reference's row
// order (src/triangle_counting/gpu_sparse_kernel.cu:25-46): the pivot is
// N+(u), the rows streamed are N+(v) for v in N+(u).  Its scratch -- the queue
// head, an error word and the total -- lives in the static words below, so the
// call allocates nothing.  At most kNoAllocMaxEdges oriented edges.
//
// What bounds it: the ids streamed (every edge streams all of N+(v)) at about
// 30 instructions per 32 ids, and on small graphs the chain of dependent loads
// of a unit.  Lanes own rows, 32 or 8 to a row, instead of searching the row
// of each id; units hold 32 to 256 edges, eight a warp, instead of 256 always;
// a unit finds its first row in 32-way steps.  B200, R-MAT s17 576 -> 289 us,
// s12 381 -> 69 us, Chung-Lu 2^17 474 -> 195 us, geometric 2^17 249 -> 129 us.
#include <algorithm>
#include <mutex>

#include "internal.h"
#include "search.cuh"

namespace bbtc {

constexpr uint64_t kNoAllocMaxEdges = 1ull << 24;  // 16,777,216 oriented edges

struct NoAllocScratch {
  uint32_t head;   // next work unit
  uint32_t error;  // bit 0: a row pointer or id outside the CSR was met
  unsigned long long total;
};

// One copy per device that loads the library, kept until the process exits.
// Host code must not take its address directly: the device address comes from
// cudaGetSymbolAddress, once per device.
static __device__ __align__(256) NoAllocScratch g_noalloc_scratch;

namespace {

constexpr uint32_t FULL = 0xffffffffu;

enum PivotKind : uint32_t { kBitmap, kList, kGlobal };

// A warp's shared memory: its buffer (bitmap or sorted list of the pivot row's
// ids), then the pivot between its build and its probes, so that the probe
// loops keep the register budget.
extern __shared__ __align__(16) uint32_t sh[];
struct Pivot {
  const uint32_t* row;
  uint32_t len;
  uint32_t base;  // bitmap bit 0 <-> id `base`
  uint32_t cap;   // a bit of the buffer that stays zero
  uint32_t first, last;
  uint32_t pad;
};
constexpr uint32_t kPivotWords = sizeof(Pivot) / 4;
static_assert(sizeof(Pivot) % 16 == 0, "the buffers stay 16-byte aligned");

// Is id x one of the pivot's?  `pos`: global kind, this lane's position of the
// last search in the same probe row.
template <uint32_t KIND>
__device__ __forceinline__ uint32_t member(uint32_t buf, const Pivot& pv, uint32_t x, uint32_t& pos) {
  if constexpr (KIND == kBitmap) {
    // ids outside the pivot's span (below base they wrap high) land on the
    // always-zero last word: no branch
    const uint32_t y = min(x - pv.base, pv.cap);
    return (sh[buf + (y >> 5)] >> (y & 31)) & 1u;
  } else if constexpr (KIND == kList) {
    if (x < pv.first || x > pv.last) return 0;
    const uint32_t p = lower_bound_u32(sh + buf, pv.len, x);
    return (p < pv.len && sh[buf + p] == x) ? 1u : 0u;
  } else {
    if (x < pv.first || x > pv.last) return 0;
    pos = gallop_lb(pv.row, pv.len, pos, x);
    return (pos < pv.len && pv.row[pos] == x) ? 1u : 0u;
  }
}

// The rows of a batch's edges (lane l holds edge l's row as start and length in
// `ids`), G lanes to a row, two rows and two steps of each in flight.
template <uint32_t KIND, uint32_t G>
__device__ __forceinline__ uint32_t probe_rows(const uint32_t* __restrict__ ids, uint32_t buf, uint32_t state,
                                               uint32_t start, uint32_t len, uint32_t cnt) {
  constexpr uint32_t E = 32 / G;  // rows side by side
  const uint32_t lane = threadIdx.x & 31;
  const Pivot pv = *reinterpret_cast<const Pivot*>(sh + state);
  uint32_t hits = 0;
  for (uint32_t r = lane / G; r < cnt + lane / G; r += 2 * E) {
    // rows past the last have length 0 (r + E never wraps: both are below 32)
    const uint32_t s0 = __shfl_sync(FULL, start, r), s1 = __shfl_sync(FULL, start, r + E);
    const uint32_t l0 = __shfl_sync(FULL, len, r), l1 = __shfl_sync(FULL, len, r + E);
    const uint32_t lm = max(l0, l1);
    uint32_t g0 = 0, g1 = 0;
    for (uint32_t i = lane & (G - 1); i < lm; i += 2 * G) {
      const bool k0 = i < l0, k1 = i < l1, k2 = i + G < l0, k3 = i + G < l1;
      uint32_t x0 = 0, x1 = 0, x2 = 0, x3 = 0;
      if (k0) x0 = __ldg(ids + s0 + i);
      if (k1) x1 = __ldg(ids + s1 + i);
      if (k2) x2 = __ldg(ids + s0 + G + i);
      if (k3) x3 = __ldg(ids + s1 + G + i);
      if (k0) hits += member<KIND>(buf, pv, x0, g0);
      if (k1) hits += member<KIND>(buf, pv, x1, g1);
      if (k2) hits += member<KIND>(buf, pv, x2, g0);
      if (k3) hits += member<KIND>(buf, pv, x3, g1);
    }
  }
  return hits;
}

// Rows of up to 32 edges against the built pivot; returns this lane's hits.
// 32 lanes to a row when rows are 20 ids or longer on average, else 8.
template <uint32_t KIND>
__device__ __noinline__ uint32_t probe(const uint32_t* ids, uint32_t buf, uint32_t state, uint32_t start,
                                       uint32_t len, uint32_t cnt) {
  const uint32_t total = __reduce_add_sync(FULL, len);
  if (total == 0) return 0;
  if (total >= 20 * cnt) return probe_rows<KIND, 32>(ids, buf, state, start, len, cnt);
  return probe_rows<KIND, 8>(ids, buf, state, start, len, cnt);
}

// Row ranges of a caller CSR, checked against [0, m] and ids against n.
struct CheckedCsrSegs {
  const uint32_t* __restrict__ col;
  const uint32_t* __restrict__ rp;
  uint32_t n;
  uint64_t m;
  uint32_t* err;
  __device__ __forceinline__ void get(uint32_t q, uint32_t& start, uint32_t& len) const {
    const uint32_t v = col[q];
    start = 0;
    len = 0;
    if (v >= n) {
      atomicOr(err, 1u);
      return;
    }
    const uint32_t a = rp[v], b = rp[v + 1];
    if (b < a || (uint64_t)b > m) {
      atomicOr(err, 1u);
      return;
    }
    start = a;
    len = b - a;
  }
};

// Edges [e, ee) of a row against the row's own ids: build, probe, clear.
template <uint32_t KIND>
__device__ __forceinline__ uint32_t pivot_pass(const uint32_t* __restrict__ prow, uint32_t pd, uint32_t base,
                                               uint32_t words, const CheckedCsrSegs& segs, uint32_t e, uint32_t ee,
                                               uint32_t buf, uint32_t state) {
  const uint32_t lane = threadIdx.x & 31;
  uint32_t* bm = sh + buf;
  if constexpr (KIND == kBitmap) {
    for (uint32_t i = lane; i < pd; i += 32) {
      const uint32_t y = prow[i] - base;
      atomicOr(&bm[y >> 5], 1u << (y & 31));
    }
  } else if constexpr (KIND == kList) {
    for (uint32_t i = lane; i < pd; i += 32) bm[i] = prow[i];
  }
  // callers keep words < the buffer size, so word `words` is never set
  if (lane == 0) *reinterpret_cast<Pivot*>(sh + state) = Pivot{prow, pd, base, words * 32, prow[0], prow[pd - 1], 0};
  __syncwarp();
  uint32_t hits = 0;
  while (e < ee) {
    const uint32_t cnt = min(32u, ee - e);
    uint32_t start = 0, len = 0;
    if (lane < cnt) segs.get(e + lane, start, len);
    hits += probe<KIND>(segs.col, buf, state, start, len, cnt);
    e += cnt;
  }
  __syncwarp();  // back to an all-zero buffer
  if constexpr (KIND == kBitmap) {
    for (uint32_t i = lane; i < words; i += 32) bm[i] = 0;
  } else if constexpr (KIND == kList) {
    for (uint32_t i = lane; i < pd; i += 32) bm[i] = 0;
  }
  __syncwarp();
  return hits;
}

// Units of `unit_edges` consecutive edges (a multiple of 32).
__global__ void __launch_bounds__(256, 4) k_count_csr_static(const uint32_t* __restrict__ indptr,
                                                             const uint32_t* __restrict__ indices, uint32_t n,
                                                             uint64_t m, uint32_t unit_edges, uint32_t units,
                                                             NoAllocScratch* scr, uint32_t bm_words) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t buf = (threadIdx.x >> 5) * (bm_words + kPivotWords), state = buf + bm_words;
  for (uint32_t i = lane; i < bm_words; i += 32) sh[buf + i] = 0;
  __syncwarp();
  const CheckedCsrSegs segs{indices, indptr, n, m, &scr->error};
  while (true) {
    uint32_t g = 0;
    if (lane == 0) g = atomicAdd(&scr->head, 1u);
    g = __shfl_sync(FULL, g, 0);
    if (g >= units) break;
    const uint32_t e0 = g * unit_edges;
    const uint64_t e1w = (uint64_t)e0 + unit_edges;
    const uint32_t e1 = (uint32_t)(e1w < m ? e1w : m);
    uint32_t e = e0;
    uint32_t u = row_of(indptr, n, e);  // < n (the host refuses n == 0 with m > 0)
    unsigned long long acc = 0;
    while (e < e1) {
      if (u >= n) {  // no row ends after e: indptr[n] < m
        if (lane == 0) atomicOr(&scr->error, 1u);
        break;
      }
      const uint32_t a = indptr[u], b = indptr[u + 1];
      if (b < a || (uint64_t)b > m || b <= e) {  // malformed row pointers: stop this unit
        if (lane == 0) atomicOr(&scr->error, 1u);
        break;
      }
      const uint32_t ee = min(b, e1);
      const uint32_t pd = b - a;
      const uint32_t* prow = indices + a;
      // the caller's row must be strictly increasing: the bitmap is indexed by id
      bool sorted = true;
      for (uint32_t i = lane; i + 1 < pd; i += 32) sorted &= prow[i] < prow[i + 1];
      if (!__all_sync(FULL, sorted)) {
        if (lane == 0) atomicOr(&scr->error, 1u);
        e = ee;
        if (e < e1) u = next_row(indptr, n, u, e, lane);
        continue;
      }
      const uint32_t first = prow[0], last = prow[pd - 1];
      const uint32_t span_words = last >= first ? ((last - first) >> 5) + 1 : 0xffffffffu;
      if (span_words < bm_words)
        acc += pivot_pass<kBitmap>(prow, pd, first, span_words, segs, e, ee, buf, state);
      else if (pd <= bm_words)
        acc += pivot_pass<kList>(prow, pd, 0, 0, segs, e, ee, buf, state);
      else
        acc += pivot_pass<kGlobal>(prow, pd, 0, 0, segs, e, ee, buf, state);
      e = ee;
      if (e < e1) u = next_row(indptr, n, u, e, lane);
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) acc += __shfl_xor_sync(FULL, acc, d);
    if (lane == 0 && acc) atomicAdd(&scr->total, acc);
  }
}

// Per device, set up by the first call on it: the device address of
// g_noalloc_scratch, the kernel's shared-memory attribute and its grid.
std::mutex g_noalloc_mu;
void* g_noalloc_ptr[kMaxDevices] = {};
uint32_t g_noalloc_grid[kMaxDevices] = {};

constexpr uint32_t kNoAllocBitmapWords = 1024, kNoAllocWarps = 8;
constexpr size_t kNoAllocSmem = (size_t)kNoAllocWarps * (kNoAllocBitmapWords + kPivotWords) * sizeof(uint32_t);

int noalloc_setup(int dev, void** ptr, uint32_t* grid) {
  std::lock_guard<std::mutex> lk(g_noalloc_mu);
  if (!g_noalloc_ptr[dev]) {
    // the device is current: resolve the array's device address
    void* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess) return cuda_fail(e, "cudaGetSymbolAddress(g_noalloc_scratch)");
    const size_t sm = kNoAllocSmem;
    BBTC_CUDA(cudaFuncSetAttribute(k_count_csr_static, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    int sms = 0, per_sm = 0;
    BBTC_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    BBTC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_count_csr_static, kNoAllocWarps * 32, sm));
    g_noalloc_grid[dev] = (uint32_t)std::max(1, sms * std::max(1, per_sm));
    g_noalloc_ptr[dev] = p;
  }
  *ptr = g_noalloc_ptr[dev];
  *grid = g_noalloc_grid[dev];
  return BBTC_OK;
}

}  // namespace

}  // namespace bbtc

extern "C" int bbtc_count_csr_noalloc(const uint32_t* d_indptr, const uint32_t* d_indices, uint32_t n, uint64_t m,
                                      uint64_t* out, void* stream) {
  using namespace bbtc;
  if (!d_indptr || (m && !d_indices) || !out) return fail(BBTC_ERR_ARG, "NULL argument");
  if (n == 0xffffffffu) return fail(BBTC_ERR_ARG, "n must be below 2^32 - 1");
  if (n == 0 && m > 0) return fail(BBTC_ERR_ARG, "a CSR with no rows cannot hold edges (n == 0, m > 0)");
  if (m > kNoAllocMaxEdges)
    return fail(BBTC_ERR_CAPACITY, "bbtc_count_csr_noalloc takes at most " + std::to_string(kNoAllocMaxEdges) +
                                       " oriented edges; got " + std::to_string(m));
  int dev = 0;
  BBTC_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= (int)kMaxDevices) return fail(BBTC_ERR_NODEV, "device index beyond the supported range");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  void* ptr = nullptr;
  uint32_t grid = 0;
  BBTC_TRY(noalloc_setup(dev, &ptr, &grid));
  NoAllocScratch* scr = static_cast<NoAllocScratch*>(ptr);
  BBTC_CUDA(cudaMemsetAsync(scr, 0, sizeof(NoAllocScratch), s));
  // about eight units a warp, so that the slow ones even out, of 32 to 256 edges: a unit builds its pivots anew
  // (R-MAT s17: 7 thousand units of 256 edges left most of the chip waiting for the last ones)
  const uint64_t share = m / ((uint64_t)grid * kNoAllocWarps * 8);
  const uint32_t unit_edges = (uint32_t)std::min<uint64_t>(256, std::max<uint64_t>(32, share & ~31ull));
  const uint32_t units = (uint32_t)((m + unit_edges - 1) / unit_edges);
  if (units > 0) {
    const size_t sm = kNoAllocSmem;
    const uint32_t blocks = std::min(grid, (units + kNoAllocWarps - 1) / kNoAllocWarps);
    k_count_csr_static<<<blocks, kNoAllocWarps * 32, sm, s>>>(d_indptr, d_indices, n, m, unit_edges, units, scr,
                                                              kNoAllocBitmapWords);
    BBTC_CUDA(cudaGetLastError());
  }
  struct {
    uint32_t head, error;
    unsigned long long total;
  } hdr{0, 0, 0};
  BBTC_CUDA(cudaMemcpyAsync(&hdr, scr, sizeof(hdr), cudaMemcpyDeviceToHost, s));
  BBTC_CUDA(cudaStreamSynchronize(s));
  if (hdr.error) return fail(BBTC_ERR_INPUT, "the CSR has a row pointer or column id outside its bounds, or an "
                                            "unsorted row");
  *out = hdr.total;
  return BBTC_OK;
}
