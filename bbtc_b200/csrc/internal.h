// Internal structures shared by the translation units of libbbtc.so.
#pragma once

#include <cuda_runtime.h>
#include <nvtx3/nvToolsExt.h>

#include <cstdint>
#include <map>
#include <memory>
#include <string>
#include <vector>

#include "../../include/bbtc_gpu.h"

namespace bbtc {

// ---- errors ---------------------------------------------------------------
void set_error(const std::string& msg);
int fail(int status, const std::string& msg);
int cuda_fail(cudaError_t e, const char* what);

#define BBTC_CUDA(call)                                   \
  do {                                                    \
    cudaError_t e__ = (call);                             \
    if (e__ != cudaSuccess) return ::bbtc::cuda_fail(e__, #call); \
  } while (0)

#define BBTC_TRY(call)          \
  do {                          \
    int rc__ = (call);          \
    if (rc__ != BBTC_OK) return rc__; \
  } while (0)

// ---- device allocations ---------------------------------------------------
// Every device allocation of the library whose failure is an error goes
// through dev_malloc / dev_malloc_sync, so that a test hook
// (bbtc_debug_fail_alloc, or BBTC_FAIL_ALLOC=k in the environment when the
// library loads) can make the k-th next one fail as if the device were out of
// memory.  take_alloc_fault() consumes the armed fault (true once, when the
// count reaches it).
bool take_alloc_fault();

template <class T>
inline cudaError_t dev_malloc(T** p, size_t bytes, cudaStream_t s) {
  if (take_alloc_fault()) {
    *p = nullptr;
    return cudaErrorMemoryAllocation;
  }
  return cudaMallocAsync(reinterpret_cast<void**>(p), bytes, s);
}

template <class T>
inline cudaError_t dev_malloc_sync(T** p, size_t bytes) {
  if (take_alloc_fault()) {
    *p = nullptr;
    return cudaErrorMemoryAllocation;
  }
  return cudaMalloc(reinterpret_cast<void**>(p), bytes);
}

// A named range on the NVTX timeline (shown by nsys, filterable in ncu with
// --nvtx); with no tool attached it costs a pointer check.
struct Range {
  explicit Range(const char* name) { nvtxRangePushA(name); }
  ~Range() { nvtxRangePop(); }
  Range(const Range&) = delete;
  Range& operator=(const Range&) = delete;
};

constexpr uint32_t kMaxParts = 64;
constexpr uint32_t kMaxDevices = 64;
constexpr uint64_t kNoSegment = ~0ull;

// One tile as the kernels see it: tile-local row pointers (H+1 entries, the
// first is 0) and tile-local column ids, both 16-byte aligned.  An empty tile
// has rp == nullptr.
struct DevTile {
  const uint32_t* rp;
  const uint32_t* col;
  const uint32_t* erow;  // row of entry 32 q, for q < ceil(nnz / 32)
  uint32_t H, W, nnz, maxdeg;
};

// Kinds of work a task is run as (see count.cu).
enum TaskKind : uint32_t {
  kPivotBitmap = 0,  // pivot row -> shared bitmap of the column part, probes test bits
  kPivotList = 1,    // pivot row -> sorted shared list, probes binary-search it
  kPivotGlobal = 2,  // pivot row too long for shared memory: binary search in global memory
};

// One queued task: `rows` is the tile whose rows are the pivot vertices and
// whose entries select the probe rows; `pivot` holds the pivot vertices' rows
// (the set each intersection is tested against) and `probe` the rows that
// are streamed against it.  For the v-centric order rows = CSC of ab
// (reversed tile (j,i)), pivot = bc, probe = ac.  For the u-centric order
// (the reference's row order) rows = ab, pivot = ac, probe = bc.
struct DevTask {
  DevTile rows;
  DevTile pivot;
  DevTile probe;
  uint32_t kind;
  uint32_t unit_edges;  // entries of `rows` per work unit
  uint32_t slot;        // output counter index
  uint32_t words;       // bitmap words the pivot part needs (ceil(W/32))
};

// One graph of a fused count: the pivot lists that the layout builds.  Entry
// q is an in-edge (u, v): rec[q] = (first, end) of the pairs of N+(u) that
// can meet N+(v).  Pivot k is 8 words: its entries [e0, e1), its row's first
// pair and number of pairs, first word, span in words, the bits kept of the
// first pair, the vertex; pivots are in entry order and end with one whose
// e0 is ~0.  crow[x] = the first pivot with entries past 32 x.
constexpr int kLevels = 5;
struct PivotGraph {
  const uint2* words;  // (32-id word, bit mask) pairs of the rows
  const uint2* rec;
  const uint4* piv;
  const uint32_t* crow;
  uint32_t entries;
  uint32_t npiv;
  uint32_t level_units[kLevels], level_size[kLevels];  // work units in queue order: counts, batches of 32 entries each
  uint32_t slot;        // output counter index
  uint32_t plain;       // 1: every pivot keeps its whole row (all bits of its first pair)
};

// A block CSR over one cut vector, for the forward or the reversed graph.
struct BlockTiles {
  uint32_t P = 0;
  std::vector<uint32_t> nnz, maxdeg, nerows;  // P*P each
  std::vector<uint64_t> rp_off, col_off;      // element offsets, kNoSegment when empty
  uint32_t* d_rp = nullptr;                    // row-pointer pool
  uint32_t* d_col = nullptr;                   // column pool
  uint32_t* d_erow = nullptr;                  // row index of every 32nd entry, per tile
  size_t rp_len = 0, col_len = 0, erow_len = 0;
  cudaStream_t stream = nullptr;
  void release(cudaStream_t s);
};

struct Plan {
  std::vector<DevTask> tasks;      // host copy: the tasks, or
  std::vector<PivotGraph> pivots;  // the graphs of a fused count
  std::vector<uint32_t> prefix;    // unit prefix, one more than items
  void* d_queue = nullptr;         // items and prefix; stream-ordered, reused while large enough
  size_t cap = 0;                  // bytes the device buffer holds
  size_t prefix_at = 0;            // byte offset of the prefix
  cudaStream_t stream = nullptr;   // stream the buffers were allocated on
  uint32_t total_units = 0;
  uint32_t launches = 0;
  bool fused = false;              // pivot lists (fused.cu)
  bool long_lists = false;         // with many in-edges per pivot
  cudaGraphExec_t exec = nullptr;
  bool captured = false;
  bool delivers = false;           // the last launch put its counts where its Delivery says
  uint32_t stage_polls = 0;        // the context's staging test hook when the launch was captured
  void release();
};

}  // namespace bbtc

struct bbtc_ctx {
  int device = 0;
  cudaStream_t stream = nullptr;
  int sms = 0;
  size_t smem_optin = 0;
  size_t smem_set = 0;                 // dynamic shared memory that the count kernels take, as far as asked
  bool open_carveout = false;          // layout kernels ask for the largest shared-memory carveout (launch_layout)
  uint32_t layout_blocks_per_sm = 8;   // grid cap of the layout kernels (256 threads a block)
  uint32_t upload_window = 0;          // host uploads: pieces in flight at most (0 = all at once)
  uint64_t zero_copy_bytes = 0;        // host arrays up to this size in mapped page-locked memory are read
                                       // by a kernel instead of the copy engines (0 = never)
  uint32_t debug_stage_polls = 0;      // test hook (bbtc_debug_stage_timeout): > 0 = staging copies are not
                                       // issued and their waits give up after this many polls
  uint32_t debug_layout_pass = 0;      // test hook (bbtc_debug_layout_timeout): the single-pass layout kernel (1 the
  uint32_t debug_layout_polls = 0;     // pairs', 2 the pivots') whose first tile stays silent, and its waits' polls
  // Page-locked staging for the small control copies (cut vectors, tile
  // offsets and statistics, counts).  A copy to or from pageable memory is
  // staged by the driver through buffers every thread shares, so one that
  // waited for a long kernel on its stream held up the copies of all other
  // threads; copies from pinned memory wait only for their own stream.
  char* h_stage = nullptr;
  uint64_t delivered = 0;  // counts delivered to h_stage (Delivery) so far; the last one is there
  bool recorded = false;   // a count was launched into a capture of the stream: its replays deliver there unseen
  // Pinned staging of the task queues' uploads, kept across plans.
  char* h_plan = nullptr;
  size_t h_plan_cap = 0;
  cudaEvent_t h_plan_done = nullptr;  // recorded after the last upload from h_plan
  cudaEvent_t ev_layout[2] = {nullptr, nullptr};  // start and end of the last layout build
  // Layout scratch kept between builds (bbtc::Scratch), at most kScratchKeep bytes.
  char* d_scratch = nullptr;
  size_t scratch_cap = 0;
};

namespace bbtc {

// Scratch of one layout build: its temporaries are carved from one device
// block that the context keeps between builds, so a build whose temporaries
// fit makes no allocation call for them.  `want` sums what the build asked
// for (256-byte rounded), carved or not; the block grows to it afterwards.
struct Scratch {
  char* base = nullptr;
  size_t cap = 0, off = 0, want = 0;
};
// The build running on this thread, if any (one build at a time per context,
// and a context's builds run on the thread that called them).
inline thread_local Scratch* t_scratch = nullptr;

// Stream-ordered device buffer (freed on the stream it was allocated on);
// carved from the running build's scratch when that has room.
struct DevBuf {
  void* p = nullptr;
  cudaStream_t s = nullptr;
  bool carved = false;
  DevBuf() = default;
  DevBuf(const DevBuf&) = delete;
  DevBuf& operator=(const DevBuf&) = delete;
  ~DevBuf() {
    if (p && !carved) cudaFreeAsync(p, s);
  }
  template <class T>
  T* as() { return static_cast<T*>(p); }
};

inline int dalloc(DevBuf& b, size_t bytes, cudaStream_t s) {
  b.s = s;
  if (Scratch* a = t_scratch) {
    const size_t need = ((bytes > 16 ? bytes : 16) + 255) & ~static_cast<size_t>(255);
    a->want += need;
    if (a->off + need <= a->cap) {
      b.p = a->base + a->off;
      b.carved = true;
      a->off += need;
      return BBTC_OK;
    }
  }
  cudaError_t e = dev_malloc(&b.p, bytes > 16 ? bytes : 16, s);
  if (e != cudaSuccess) {
    cudaGetLastError();
    b.p = nullptr;
    return fail(BBTC_ERR_NOMEM, std::string("device allocation of ") + std::to_string(bytes) +
                                    " bytes failed: " + cudaGetErrorString(e));
  }
  return BBTC_OK;
}

constexpr uint32_t kCountWords = 6;  // of bbtc_graph::d_count

// Regions of bbtc_ctx::h_stage (one graph build or count at a time per context).
constexpr size_t kStageBytes = 1u << 20;
constexpr size_t kStageCuts = 0;          // cut vector, <= (64 + 2) x 4 bytes
constexpr size_t kStageFlags = 3072;      // contract flags and totals of a layout build; small read-backs
constexpr size_t kStageCount = 3584;      // the last delivered count and its control word
constexpr size_t kStageOff[2] = {4096, 40960};      // tile offsets of the block CSRs (<= 32,768 bytes each)
constexpr size_t kStageStats[2] = {81920, 163840};  // their tile statistics (<= 81,920 bytes each)
constexpr size_t kStageOut = 262144;      // counts read back (<= 98,304 of them)

}  // namespace bbtc

struct bbtc_graph {
  bbtc_ctx* ctx = nullptr;
  uint32_t n = 0, P = 0;
  uint64_t m = 0;
  std::vector<uint32_t> cuts;
  uint32_t* d_indptr = nullptr;   // resident oriented CSR (global ids)
  uint32_t* d_indices = nullptr;
  void* d_words = nullptr;        // word-compressed rows: (word, mask) uint2 pairs
  uint64_t nwords = 0;            // pairs
  void* d_rec = nullptr;          // pivot lists (PivotGraph): one uint2 per in-edge
  void* d_piv = nullptr;          // npiv + 1 pivots of 32 bytes
  uint32_t* d_crow = nullptr;     // pivot of every 32nd entry
  uint32_t npiv = 0;
  uint64_t nentry_rows = 0;       // words of d_crow
  uint32_t sparse_end = 0;        // 32-entry batches up to which pivots have few in-edges
  bool oriented = false;          // every id exceeds its row's
  bbtc::BlockTiles fwd, rev;      // tiles of the per-task kernels, built on first use
  uint64_t* d_count = nullptr;  // kCountWords: a count and its control word; then a queue kernel's accumulators
  uint64_t delivered = 0;       // which of the context's delivered counts the last one is, 0 = none
  uint64_t device_bytes = 0;
  double layout_ms = 0;
  bool fwd_built = false;         // the forward block CSR is built on first use (task-list counting, tile stats)
  bool rev_built = false;         // the reversed one too (v-centric task-list counting)
  bool zero_copy = false;         // the upload read the host CSR with a kernel (no copy-engine transfer)
  uint32_t last_launches = 0;
  std::map<std::string, std::unique_ptr<bbtc::Plan>> plans;  // cached queues keyed by request
};

namespace bbtc {

// layout.cu
// indptr / indices are host memory when `host`, else device memory of the
// context's device; the graph keeps its own device copy either way.
int build_layout(bbtc_graph* g, const uint32_t* indptr, const uint32_t* indices, bool host);
// Build g's forward block CSR if it is not built yet (on g's context stream; synchronises it).
int ensure_fwd(bbtc_graph* g);
// The same for both block CSRs.
int ensure_tiles(bbtc_graph* g);
DevTile dev_tile(const BlockTiles& t, const std::vector<uint32_t>& cuts, uint32_t x, uint32_t y);

// Where a queue kernel's last warp writes the counts (deliver.cuh): `host`
// (page-locked) and, unless NULL, `dev`, each with the control word after the
// counts.  `acc` is what the warps add to, kDeliverWords longer than the
// counts; it is zero before the launch and again after it.
constexpr uint32_t kDeliverWords = 2;
struct Delivery {
  uint64_t* acc = nullptr;
  uint64_t* dev = nullptr;
  uint64_t* host = nullptr;
};

// count.cu
// With a Delivery, a queue of at least one unit puts its counts there instead
// of d_outs (plan->delivers), which saves the clearing and the copy.
int count_enqueue(bbtc_ctx* ctx, const std::vector<bbtc_graph*>& graphs,
                  const std::vector<std::vector<bbtc_task>>& tasks, const bbtc_opts& o, bool fused,
                  uint64_t* d_outs, Plan* plan, bool reuse, const Delivery* to = nullptr);
int kernel_smem_optin(bbtc_ctx* ctx, const bbtc_opts& o);
// Every launch of count_enqueue leaves a control word after its counts
// (d_outs[graphs.size()]): BBTC_ERR_TIMEOUT if a shared-memory staging copy
// gave up waiting (the counts are void).
int control_status(uint64_t ctrl);
size_t smem_bytes_for(const bbtc_opts& o);

// Options shared by the count kernels.
inline uint32_t norm_bm_words(uint32_t w) {
  if (w == 0) w = 1024;
  w = (w + 3) & ~3u;
  return w < 256 ? 256 : w;
}
inline uint32_t norm_warps(uint32_t w) { return w == 0 || w > 8 ? 8 : w; }

// fused.cu
size_t pivots_smem(uint32_t bm_words, uint32_t warps);
int pivots_smem_optin(size_t bytes);
int pivots_launch(bbtc_ctx* ctx, const PivotGraph& one, const PivotGraph* d_many, const uint32_t* d_prefix, uint32_t ng,
                  uint32_t total_units, bool long_lists, const bbtc_opts& o, uint64_t* d_outs, uint32_t nouts,
                  uint64_t* dev, uint64_t* host);

}  // namespace bbtc
