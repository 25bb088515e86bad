// Exact subgraph enumeration: candidate filtering + worst-case-optimal-join
// extension by sorted-list intersection, as a memory-bounded hybrid
// BFS/DFS over level tables.
//
// Replaces the reference GPU WOJ path (WOJFilterVCKernel
// core/task/gpu_task/kernel/kernel_woj_subsio.cu:532-604, the per-table
// MergeSort core/task/gpu_task/kernel/algorithms/sort.cuh:59-105 and
// WOJJoinKernel kernel_woj_subsio.cu:623-721), which joins one key column at
// a time, never checks cycle closure or injectivity and caps its output at
// kMaxNumWeft rows.  Here:
//   * a level table holds partial matches of prefix length i (SoA columns);
//   * the work kernel picks, per row, the shortest label slice among the
//     backward neighbours' adjacency (the driving list) and the scan turns
//     the driving lengths into an element index space;
//   * the expand kernel deals that space to warps in tasks of consecutive
//     elements (row, driving entry), so hub rows spread over many warps; the
//     other backward slices are probed in the hub bitmap when their vertex is
//     a hub, else by binary search, injectivity is checked against the row,
//     and the survivors of a task are filtered (label, degree, neighbour
//     labels) and appended with one atomic (__ballot_sync / __popc ranks);
//   * the levels of a call are queued at once with their sizes on the device; a
//     level that does not fit its table stops the chain, and the host grows the
//     table or walks on from there depth-first, expanding at most `cap` elements
//     of a level before descending, so intermediate results never exceed the
//     scratch budget;
//   * in count mode the last position is never materialised: when it has a
//     single backward neighbour its count is the slice length minus the
//     injectivity collisions, added while expanding the position before it;
//     a two-position pendant tail is counted from a table of two-hop aggregates
//     while expanding the position three before the end.
#include <algorithm>
#include <cstring>
#include <memory>
#include <numeric>
#include <type_traits>

#include "mg_device.cuh"
#include "mg_limits.h"
#include "mg_row_sort.cuh"

namespace mg {

const char* last_error_cstr();

// ---------------------------------------------------------------------------
// Workspace (per graph handle)
// ---------------------------------------------------------------------------
// Pendant-tail keys of a call and their tables of two-hop aggregates.
struct TailStore {
  uint4* agg = nullptr;
  uint64_t cap = 0;
  TailKey* keys = nullptr;
  uint32_t keys_cap = 0;
  void free() {
    cudaFree(agg);
    cudaFree(keys);
    agg = nullptr;
    keys = nullptr;
    cap = keys_cap = 0;
  }
};

struct Workspace {
  // Level tables: rows[l] rows of prefix length l, all arrays of a level in one
  // block; they grow when a call needs more (ensure_level).
  uint64_t rows[MAXK] = {};
  void* block[MAXK] = {};
  uint32_t* col[MAXK][MAXK] = {};
  uint32_t* qid[MAXK] = {};
  uint64_t* woff[MAXK] = {};
  uint32_t* dstart[MAXK] = {};
  uint8_t* dci[MAXK] = {};
  uint32_t* tile_row = nullptr;  // first row of every expand tile of a segment
  unsigned long long* status = nullptr;  // look-back words of the work/scan kernel
  uint64_t status_bytes = 0;
  uint32_t epoch = 0;
  uint32_t* root_keep = nullptr; // matrix-filter keep bits of the level-0 candidates
  uint64_t root_keep_words = 0;
  TailStore tails;
  // Results of a call of nq queries, one block: counters (C_NUM), counts (nq),
  // rows per prefix length (nq * (MAXK + 1)), elements scheduled (nq).
  unsigned long long* res = nullptr;
  PlanDev* plans = nullptr;
  uint32_t nq_cap = 0;                   // queries that res and plans hold
  // Pinned: one plan, and a mirror of one query's result block.
  PlanDev* h_plan = nullptr;
  unsigned long long* h_res = nullptr;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr, ev2 = nullptr, ev3 = nullptr;
};

// Counter slots.  A level's slots lie together, so that clearing everything
// from a level on is one memset.
enum : int {
  C_BALG = 0, C_BALGC = 1, C_ERR = 2, C_EMIT = 3,
  C_LVL = 4,                    // slots of level l from C_LVL + 4 * l on:
  L_OUT = 0,                    // rows the expand of level l wrote (= rows of level l+1)
  L_TILE = 1,                   // work-queue position of the expand of level l
  L_T = 2,                      // candidate elements of level l
  L_SCAN = 3,                   // tile counter of the work/scan kernel of level l
  C_STOP = C_LVL + 4 * MAXK,    // 1 + the level whose elements passed their limit
  C_NUM
};
constexpr int lvl_slot(int l, int what) { return C_LVL + 4 * l + what; }

void free_workspace(Workspace* ws) {
  if (!ws) return;
  for (void* p : ws->block) cudaFree(p);
  for (void* p : {(void*)ws->tile_row, (void*)ws->status, (void*)ws->root_keep, (void*)ws->res,
                  (void*)ws->plans})
    cudaFree(p);
  ws->tails.free();
  if (ws->h_plan) cudaFreeHost(ws->h_plan);
  for (cudaEvent_t e : {ws->ev0, ws->ev1, ws->ev2, ws->ev3})
    if (e) cudaEventDestroy(e);
  delete ws;
}

// Replaces *p by `bytes` of device memory (contents are lost).
static int ws_alloc(void** p, size_t bytes) {
  cudaFree(*p);
  *p = nullptr;
  const cudaError_t e = cudaMalloc(p, std::max<size_t>(bytes, 16));
  if (e == cudaSuccess) return MG_OK;
  cudaGetLastError();
  *p = nullptr;
  return set_error(MG_E_OOM, "enumeration scratch: cudaMalloc(%zu) failed: %s", bytes,
                   cudaGetErrorString(e));
}

constexpr uint64_t kDefaultCap = 1ull << 24;
constexpr uint32_t kProbeMin = 1;  // default: every hub slice is probed in the bitmap
constexpr int EXPAND_BLOCK = 256;
constexpr int EXPAND_TILE = 1024;                 // elements per expand tile
constexpr int XSTAGE = 256;                       // survivors a warp stages at a time
constexpr uint64_t kSegment = 1ull << 30;         // elements per expand launch
constexpr int WS_ROWS = 1024;                     // rows per work/scan tile (4 per thread)
constexpr uint32_t kSpinLimit = 1u << 22;         // polls of a look-back wait (~0.3 s)
// Words of the result block of nq queries.
constexpr uint64_t res_words(uint64_t nq) { return C_NUM + nq * (MAXK + 3); }

static uint64_t level_row_bytes(int l) { return uint64_t(l) * 4 + 4 + 4 + 8 + 4 + 1; }

// Rows that a level table starts with.  Tables for 2^24 rows at once (the most
// a level holds by default) cost 2 GB and 12 ms of allocation in a graph's first
// calls and 10 ms when it is freed; most queries need a small part of them.
constexpr uint64_t kFirstRows = 1ull << 17;

// Makes room for `rows` rows of prefix length l (the table's contents are lost).
static int ensure_level(Workspace* ws, int l, uint64_t rows) {
  if (ws->rows[l] >= rows) return MG_OK;
  auto pad = [](uint64_t b) { return (b + 255) & ~uint64_t(255); };
  const uint64_t words = pad(rows * 4), offs = pad((rows + 1) * 8);
  ws->rows[l] = 0;
  int rc = ws_alloc(&ws->block[l], words * (l + 2) + offs + pad(rows));
  if (rc) return rc;
  auto* p = static_cast<unsigned char*>(ws->block[l]);
  auto take = [&](uint64_t bytes) {
    unsigned char* q = p;
    p += bytes;
    return q;
  };
  for (int j = 0; j < l; ++j) ws->col[l][j] = reinterpret_cast<uint32_t*>(take(words));
  ws->qid[l] = reinterpret_cast<uint32_t*>(take(words));
  ws->dstart[l] = reinterpret_cast<uint32_t*>(take(words));
  ws->woff[l] = reinterpret_cast<uint64_t*>(take(offs));
  ws->dci[l] = take(pad(rows));
  ws->rows[l] = rows;
  return MG_OK;
}

// Scratch of a walk with level tables of at most `cap` rows for nq queries.
static int ensure_ws(DevGraph* dg, uint64_t cap, uint32_t nq) {
  int rc;
  if (!dg->ws) {
    // Built aside: the graph never keeps a workspace that is not complete.
    std::unique_ptr<Workspace, void (*)(Workspace*)> made(new Workspace(), free_workspace);
    static_assert(sizeof(PlanDev) % 8 == 0, "the result block follows the plan");
    MG_CK(cudaMallocHost((void**)&made->h_plan, sizeof(PlanDev) + res_words(1) * 8));
    made->h_res = reinterpret_cast<unsigned long long*>(made->h_plan + 1);
    for (cudaEvent_t* e : {&made->ev0, &made->ev1, &made->ev2, &made->ev3})
      MG_CK(cudaEventCreate(e));
    if ((rc = ws_alloc((void**)&made->tile_row, (kSegment / EXPAND_TILE + 2) * 4))) return rc;
    dg->ws = made.release();
  }
  Workspace* ws = dg->ws;
  const uint64_t status = (std::max<uint64_t>(cap, nq) / WS_ROWS + 2) * 8;
  if (ws->status_bytes < status) {
    ws->status_bytes = 0;
    if ((rc = ws_alloc((void**)&ws->status, status))) return rc;
    MG_CK(cudaMemsetAsync(ws->status, 0, status, dg->stream));
    ws->status_bytes = status;
    ws->epoch = 0;
  }
  if (ws->nq_cap < nq) {
    ws->nq_cap = 0;
    if ((rc = ws_alloc((void**)&ws->res, res_words(nq) * 8))) return rc;
    if ((rc = ws_alloc((void**)&ws->plans, uint64_t(nq) * sizeof(PlanDev)))) return rc;
    ws->nq_cap = nq;
  }
  return MG_OK;
}

// ---------------------------------------------------------------------------
// Kernels
// ---------------------------------------------------------------------------
struct TabPtrs {
  uint32_t* col[MAXK];
  uint32_t* qid;  // nullptr: single query, q = 0
};

struct StepArgs {
  GraphDev g;
  const PlanDev* plans;
  uint32_t level;   // rows hold positions 0..level-1; position `level` is extended
  uint32_t R;       // rows of the input table (level 0)
  TabPtrs in;
  uint64_t* woff;
  uint32_t* dstart;
  uint8_t* dci;
  uint64_t t0, t1;  // element range of this expand launch
  TabPtrs out;
  uint64_t out_cap;
  unsigned long long* ctr;
  unsigned long long* counts;
  unsigned long long* lvl_rows;  // per query: surviving prefixes of length 0..MAXK
  unsigned long long* q_elems;   // per query: candidate elements scheduled so far
  unsigned long long q_budget;   // per-query element budget (0: none)
  uint32_t count_mode;
  uint32_t filters;
  uint32_t nq;
  uint32_t* emit_col[MAXK];  // emitted rows by column,
  unsigned long long* emit_key;  // or packed: the id of query vertex u is emit_bits bits
  uint32_t emit_k, emit_bits;    // from bit (emit_k - 1 - u) * emit_bits on
  uint64_t emit_cap;
  uint64_t root_begin, root_end;  // level-0 candidate range (root_end 0: all)
  uint32_t root_step;             // level-0 stride inside the range (>= 1)
  uint32_t probe_min;             // shortest hub slice probed in the hub bitmap
  uint32_t* tile_row;              // first row of each tile of [t0, t1)
  uint32_t grab;   // expand tiles taken per work-queue grab
  const TailKey* tkeys;
  // Two-position pendant tails (tail_dense): counted while expanding
  // position k-3; the two-hop aggregates of m_p are read at
  // tail_agg[tkeys[kid].base + m_p - tkeys[kid].b0].
  uint32_t tail_dense;
  uint32_t star;  // two-leaf star endings are counted in closed form (PlanDev::star2)
  const uint4* tail_agg;
  // Level 0 of a single query is one row that needs no table: its candidates
  // are root_first + e * root_step, e < T0.
  uint64_t T0;
  uint32_t root_first;
  // Sizes on the device: row and element counts come from the level's counter
  // slots and no host value of R, t0 or t1 is read.  lane: a batch lane, whose
  // query is counted again when it does not fit.
  uint32_t dev, lane;
  uint32_t out_slot, tile_slot;  // counter slots of the output rows / work queue
  uint64_t cap_rows;             // rows of a level table
  uint64_t t_limit;              // a level with more elements stops the walk
  uint64_t seg_cap;              // elements the tile-row table covers
  unsigned long long* scan_status;  // look-back words of the work/scan kernel
  uint32_t spin_limit;           // bounded device waits (iterations)
  const uint32_t* root_keep;     // level-0 candidates kept by the matrix filter
                                 // (bit per vertex; nullptr: no filter)
};

// Kernels of a chain are launched as programmatic dependents: one may begin
// before the kernel ahead of it has ended, and waits here before it reads
// anything of it.  What a kernel of the chain writes (level tables, woff,
// tile_row, counters) is read with ordinary loads only: the wait orders those,
// while __ldg is for data that does not change while the kernel is resident,
// which here are the graph's arrays and what was finished before the chain
// began (tail tables, keep bits).
__device__ __forceinline__ void chain_begin() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Rows of the input table of a launch with sizes on the device.
__device__ __forceinline__ uint64_t dev_rows(const StepArgs& a) {
  if (a.level == 0) return a.R;
  const uint64_t r = a.ctr[lvl_slot(int(a.level) - 1, L_OUT)];
  return r < a.cap_rows ? r : a.cap_rows;
}

__device__ __forceinline__ uint32_t lanemask_lt() {
  uint32_t l = threadIdx.x & 31;
  return (1u << l) - 1u;
}

// Binary search for x in the sorted range a[s, e).
__device__ __forceinline__ bool contains(const uint32_t* __restrict__ a, uint32_t s, uint32_t e,
                                         uint32_t x) {
  uint32_t lo = s, hi = e;
  while (lo < hi) {
    uint32_t mid = (lo + hi) >> 1;
    uint32_t v = __ldg(a + mid);
    if (v < x) lo = mid + 1;
    else hi = mid;
  }
  return lo < e && __ldg(a + lo) == x;
}

__device__ __forceinline__ void slice_of(const GraphDev& g, uint32_t dir, uint32_t y,
                                         uint32_t lab, uint32_t& s, uint32_t& e) {
  const uint32_t* p = g.loff[dir] + uint64_t(lab) * g.n + y;
  s = __ldg(p);
  e = __ldg(p + 1);
}

// Probe strategy: a slice of a hub with at least `pmin` entries is probed in
// the hub's bitmap (one load, but a random sector of a row that may not sit
// in L2); shorter slices and non-hubs by binary search (a few loads that
// usually hit L1, since the elements of one row probe the same slice).
__device__ __forceinline__ bool hub_bit(const GraphDev& g, uint32_t d, uint16_t h, uint32_t x) {
  return (__ldg(g.hub_bits[d] + uint64_t(h) * g.hub_words + (x >> 5)) >> (x & 31)) & 1u;
}

// x in the d-adjacency of y, where x is known to carry the label of the slice
// [s, e) of y being asked about.
__device__ __forceinline__ bool in_slice_se(const GraphDev& g, uint32_t d, uint32_t y, uint32_t s,
                                            uint32_t e, uint32_t x, uint32_t pmin) {
  if (g.hub_slot[d] && e - s >= pmin) {
    const uint16_t h = __ldg(g.hub_slot[d] + y);
    if (h != NO_HUB) return hub_bit(g, d, h, x);
  }
  return contains(g.adj[d], s, e, x);
}

// x (labelled lab) in the label-lab slice of y's d-adjacency; with pmin <= 1
// a hub needs no slice offsets at all.
__device__ __forceinline__ bool in_slice(const GraphDev& g, uint32_t d, uint32_t y, uint32_t lab,
                                         uint32_t x, uint32_t pmin) {
  uint32_t s, e;
  if (g.hub_slot[d] && pmin <= 1) {
    const uint16_t h = __ldg(g.hub_slot[d] + y);
    if (h != NO_HUB) return hub_bit(g, d, h, x);
    slice_of(g, d, y, lab, s, e);  // not a hub: search the slice
    return contains(g.adj[d], s, e, x);
  }
  slice_of(g, d, y, lab, s, e);
  return in_slice_se(g, d, y, s, e, x, pmin);
}

__device__ __forceinline__ bool pass_filters(const GraphDev& g, const PlanDev& P, uint32_t i,
                                             uint32_t x, uint32_t filters) {
  if (filters & MG_FILTER_DEGREE) {
    if (__ldg(g.deg[0] + x) < P.req[0][i]) return false;
    if (!g.symmetric && __ldg(g.deg[1] + x) < P.req[1][i]) return false;
  }
  if (filters & MG_FILTER_NLB) {
    for (uint32_t w = 0; w < g.W; ++w) {
      if (P.nlbq[0][i][w] & ~__ldg(g.nlb[0] + uint64_t(x) * g.W + w)) return false;
      if (!g.symmetric && (P.nlbq[1][i][w] & ~__ldg(g.nlb[1] + uint64_t(x) * g.W + w)))
        return false;
    }
  }
  return true;
}

__device__ __forceinline__ bool has_self(const GraphDev& g, uint32_t x) {
  return (__ldg(g.selfbits + (x >> 5)) >> (x & 31)) & 1u;
}

__device__ __forceinline__ unsigned long long warp_sum(unsigned long long v) {
  for (int d = 16; d > 0; d >>= 1) v += __shfl_down_sync(FULL, v, d);
  return v;
}

// Largest r in [lo, hi] with woff[r] <= t (woff non-decreasing, woff[lo] <= t).
__device__ __forceinline__ uint32_t find_row(const uint64_t* woff, uint32_t lo, uint32_t hi,
                                             uint64_t t) {
  while (lo < hi) {
    uint32_t mid = (lo + hi + 1) >> 1;
    if (woff[mid] <= t) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// Adds a thread's accumulated match count and prefix survivors of query q:
// s1 prefixes of length i+1, s2 of length i+2 and sk of length k (the last
// two from closed-form counts).
__device__ __forceinline__ void acc_flush(const StepArgs& a, uint32_t q, uint32_t i,
                                          unsigned long long cnt, unsigned long long s1,
                                          unsigned long long sk, unsigned long long s2 = 0) {
  if (cnt) atomicAdd(&a.counts[q], cnt);
  unsigned long long* L = a.lvl_rows + uint64_t(q) * (MAXK + 1);
  if (s1) atomicAdd(&L[i + 1], s1);
  if (s2) atomicAdd(&L[i + 2], s2);
  if (sk) atomicAdd(&L[a.plans[q].k], sk);
}

// Flush of a warp's accumulators: one atomic per value when every lane holds
// the same query, else one per lane.
__device__ __forceinline__ void acc_flush_warp(const StepArgs& a, uint32_t q, uint32_t i,
                                               unsigned long long& cnt,
                                               unsigned long long& s1,
                                               unsigned long long& sk,
                                               unsigned long long& s2, bool force) {
  const bool uniform = __all_sync(FULL, q == __shfl_sync(FULL, q, 0));
  if (uniform) {
    const unsigned long long c = warp_sum(cnt), x = warp_sum(s1), y = warp_sum(sk),
                             z = warp_sum(s2);
    if ((threadIdx.x & 31) == 0) acc_flush(a, q, i, c, x, y, z);
    cnt = s1 = sk = s2 = 0;
  } else if (force) {
    acc_flush(a, q, i, cnt, s1, sk, s2);
    cnt = s1 = sk = s2 = 0;
  }
}

// Two-hop aggregates of the tail keys, for every vertex y of label lp:
//   A(y)  = sum_{x in N^{da}_{la}(y)} (|N^{db}_{lb}(x)| - [x self-loop, la == lb]),
//   AD(y) = sum_{x in N^{da}_{la}(y)} |N^{db}_{lb}(x)|
// as {A, AD, |N^{da}_{la}(y)|, degree of y}: all that closing a tail at y reads is
// one 16-byte load.  (The x of a sum are distinct vertices, so sums are below the
// number of adjacency entries, 2^32.)
// A block takes TA_V vertices of one key's bucket: short slices by a thread
// each, longer ones by a warp, the longest by the block (hubs come first in a
// bucket).  The slices of a block are one range of adj and their lengths come
// from one label's offsets, so a table costs a pass over the edges between two
// labels.  Tables for hubs only, a key per launch and a warp per hub, took 27
// launches and 2.4 ms in a batch of 64 queries, and the other vertices' sums
// were filled in by whichever candidate came first.
constexpr int TA_BLOCK = 256, TA_V = 256;
constexpr uint32_t TA_WARP = 16, TA_ALL = 2048;  // slices above: a warp each, the block

__global__ void __launch_bounds__(TA_BLOCK) k_tail_table(GraphDev g, const TailKey* keys,
                                                         uint4* agg) {
  const TailKey tk = keys[blockIdx.y];
  const uint32_t b1 = __ldg(g.bucket_off + tk.lp + 1), lane = threadIdx.x & 31;
  const uint64_t v0 = tk.b0 + uint64_t(blockIdx.x) * TA_V;
  if (tk.base == ~0ull || v0 >= b1) return;
  const uint32_t nv = min(uint32_t(TA_V), uint32_t(b1 - v0));
  uint4* out = agg + tk.base + (v0 - tk.b0);
  auto put = [&](uint32_t at, unsigned long long a, unsigned long long d, uint32_t len) {
    out[at] = make_uint4(uint32_t(a), uint32_t(d), len, __ldg(g.deg[0] + v0 + at));
  };
  __shared__ uint32_t s_long[TA_V], s_all[TA_V], n_long, n_all;
  __shared__ unsigned long long s_a, s_d;
  if (threadIdx.x == 0) n_long = n_all = 0;
  __syncthreads();
  auto sum = [&](uint32_t s, uint32_t e, uint32_t at, uint32_t step, unsigned long long& a,
                 unsigned long long& d) {
    for (uint32_t q = s + at; q < e; q += step) {
      const uint32_t x = __ldg(g.adj[tk.da] + q);
      uint32_t xs, xe;
      slice_of(g, tk.db, x, tk.lb, xs, xe);
      d += xe - xs;
      a += xe - xs - ((tk.la == tk.lb && has_self(g, x)) ? 1u : 0u);
    }
  };
  uint32_t s = 0, e = 0;
  if (threadIdx.x < nv) {
    slice_of(g, tk.da, uint32_t(v0) + threadIdx.x, tk.la, s, e);
    if (e - s <= TA_WARP) {
      unsigned long long a = 0, d = 0;
      sum(s, e, 0, 1, a, d);
      put(threadIdx.x, a, d, e - s);
    } else if (e - s <= TA_ALL) {
      s_long[atomicAdd(&n_long, 1u)] = threadIdx.x;
    } else {
      s_all[atomicAdd(&n_all, 1u)] = threadIdx.x;
    }
  }
  __syncthreads();
  for (uint32_t j = threadIdx.x >> 5; j < n_long; j += TA_BLOCK / 32) {
    unsigned long long a = 0, d = 0;
    slice_of(g, tk.da, uint32_t(v0) + s_long[j], tk.la, s, e);
    sum(s, e, lane, 32, a, d);
    a = warp_sum(a);
    d = warp_sum(d);
    if (lane == 0) put(s_long[j], a, d, e - s);
  }
  for (uint32_t j = 0; j < n_all; ++j) {
    if (threadIdx.x == 0) s_a = s_d = 0;
    __syncthreads();
    unsigned long long a = 0, d = 0;
    slice_of(g, tk.da, uint32_t(v0) + s_all[j], tk.la, s, e);
    sum(s, e, threadIdx.x, TA_BLOCK, a, d);
    a = warp_sum(a);
    d = warp_sum(d);
    if (lane == 0) {
      atomicAdd(&s_a, a);
      atomicAdd(&s_d, d);
    }
    __syncthreads();
    if (threadIdx.x == 0) put(s_all[j], s_a, s_d, e - s);
    __syncthreads();
  }
}

// Table entry of m_p (see k_tail_table): read from the key's table, or summed
// over the label-l_a slice of m_p when the key has none.
__device__ __forceinline__ uint4 tail_entry(const StepArgs& a, const PlanDev& P, uint32_t mp) {
  const GraphDev& g = a.g;
  const TailKey& tk = a.tkeys[P.tail_kid];
  const uint64_t base = tk.base;
  if (base != ~0ull) return __ldg(a.tail_agg + base + (mp - tk.b0));
  const uint32_t la = tk.la, lb = tk.lb;
  uint32_t s, e, c = 0, d = 0;
  slice_of(g, P.tail_da, mp, la, s, e);
  for (uint32_t j = s; j < e; ++j) {
    const uint32_t x = __ldg(g.adj[P.tail_da] + j);
    uint32_t xs, xe;
    slice_of(g, P.tail_db, x, lb, xs, xe);
    d += xe - xs;
    c += xe - xs - ((la == lb && has_self(g, x)) ? 1u : 0u);
  }
  return make_uint4(c, d, e - s, __ldg(g.deg[0] + mp));
}

// z in the slice [s, e) of y's d-adjacency (z carries that slice's label), where
// y, of label ylab, is the candidate at hand (`cur`) or a vertex of its row and
// z a vertex of the row.  In a symmetric graph the question is put to the row's
// vertex, whose hub row or slice all candidates of the row share.
__device__ __forceinline__ bool joined(const StepArgs& a, uint32_t d, uint32_t y, uint32_t ylab,
                                       bool cur, uint32_t s, uint32_t e, uint32_t z) {
  if (cur && z != y && a.g.symmetric) return in_slice(a.g, d, z, ylab, y, a.probe_min);
  return in_slice_se(a.g, d, y, s, e, z, a.probe_min);
}

// Closed-form count of one prefix of length a = k-2 under a two-position
// pendant tail (PlanDev::tail2).  With I the matched prefix, S = the
// label-l_a slice [s, e) of m_p, D(x) = |N_{l_b}(x)| and c(x) = D(x) - [x has
// a self-loop and l_a == l_b], and A(y) = sum_{x in S(y)} c(x),
// AD(y) = sum_{x in S(y)} D(x):
//   count = A(m_p) - sum_{i in Ia, m_i in S} (c(m_i) - #{j in J : m_j in N_{l_b}(m_i)})
//           - sum_{j in J} |S|                   (every j in J is p itself)
// Also returns the number of length-(k-1) prefixes |S \ I| and their
// algorithmic bytes sum_{x in S \ I} D(x).  col(j) is the vertex matched at
// position j < a.
template <class Col>
__device__ __forceinline__ void tail_close(const StepArgs& a, const PlanDev& P, Col col,
                                           uint32_t Ia, uint32_t mp, bool cur,
                                           const uint4& entry, unsigned long long& cnt,
                                           unsigned long long& pre, unsigned long long& dsum) {
  const GraphDev& g = a.g;
  const uint32_t ia = P.k - 2;
  const uint32_t la = P.label[ia], lb = P.label[ia + 1];
  const uint32_t da = P.tail_da, db = P.tail_db;
  long long c = entry.x, d = entry.y;
  unsigned long long inS = 0;
  for (uint32_t mi = Ia; mi; mi &= mi - 1) {
    const uint32_t i2 = __ffs(mi) - 1;
    const uint32_t x = col(i2);
    bool in;
    if (cur && x != mp && g.symmetric) {  // asked of the row's vertex (see joined)
      in = in_slice(g, da, x, P.label[P.tail_p], mp, a.probe_min);
    } else {
      in = in_slice(g, da, mp, la, x, a.probe_min);
    }
    if (!in) continue;
    inS += 1;
    uint32_t xs, xe;
    slice_of(g, db, x, lb, xs, xe);
    long long cx = (long long)(xe - xs);
    d -= cx;
    if (la == lb && has_self(g, x)) cx -= 1;
    for (uint32_t mj = P.tail_J; mj; mj &= mj - 1) {
      const uint32_t j = __ffs(mj) - 1;
      if (in_slice_se(g, db, x, xs, xe, col(j), a.probe_min)) cx -= 1;
    }
    c -= cx;
  }
  c -= (long long)__popc(P.tail_J) * (long long)entry.z;
  cnt = (unsigned long long)c;
  pre = (unsigned long long)entry.z - inS;
  dsum = (unsigned long long)d;
}

// Closed-form count of one prefix of length k-2 whose plan ends in two leaves
// a = k-2, b = k-1 of one anchor p (PlanDev::star2).  S_a and S_b are the
// label-l_a and label-l_b slices of m_p in direction d; A_x is |S_x| minus the
// earlier matches labelled l_x that lie in S_x (injectivity).  Then
//   count = A_a * (A_a - 1)   when l_a == l_b (S_b == S_a, b differs from a),
//   count = A_a * A_b         otherwise (a and b cannot collide),
// the prefixes of length k-1 number A_a, and the algorithmic bytes of the two
// positions are (8 + 4|S_a|) per prefix of length k-2 plus (8 + 4|S_b|) per
// prefix of length k-1 (count-mode definition: 8 for the last position).
// col(j) is the vertex matched at position j < k-2.
template <class Col>
__device__ __forceinline__ void star_close(const StepArgs& a, const PlanDev& P, Col col, bool cur,
                                           unsigned long long& cnt, unsigned long long& pre,
                                           unsigned long long& bal,
                                           unsigned long long& balc) {
  const GraphDev& g = a.g;
  const uint32_t ia = P.k - 2, ib = P.k - 1, d = P.star_d;
  const uint32_t mp = col(P.star_p);
  uint32_t sa, ea;
  slice_of(g, d, mp, P.label[ia], sa, ea);
  unsigned long long A = ea - sa;
  for (uint32_t m = P.samelab[ia]; m; m &= m - 1)
    if (joined(a, d, mp, P.label[P.star_p], cur, sa, ea, col(__ffs(m) - 1))) A -= 1;
  unsigned long long lb_len;
  if (P.label[ib] == P.label[ia]) {
    cnt = A ? A * (A - 1) : 0ull;
    lb_len = ea - sa;
  } else {
    uint32_t sb, eb;
    slice_of(g, d, mp, P.label[ib], sb, eb);
    unsigned long long B = eb - sb;
    for (uint32_t m = P.samelab[ib]; m; m &= m - 1)
      if (joined(a, d, mp, P.label[P.star_p], cur, sb, eb, col(__ffs(m) - 1))) B -= 1;
    cnt = A * B;
    lb_len = eb - sb;
  }
  pre = A;
  bal = 8ull + 4ull * (ea - sa) + A * (8ull + 4ull * lb_len);
  balc = 8ull + 4ull * (ea - sa) + A * 8ull;
}

// Driving slice of table row r at position a.level: its length (the row's
// candidate elements, 0 when nothing is to be expanded), start and constraint
// index (DCI_BUCKET: the label bucket), and the row's algorithmic-byte
// charges (full-slice and count-mode definitions).
__device__ __forceinline__ uint32_t row_work(const StepArgs& a, const PlanDev& P, uint64_t r,
                                             uint32_t q, uint32_t& bs, uint8_t& bci,
                                             unsigned long long& ch, unsigned long long& chc) {
  const GraphDev& g = a.g;
  const uint32_t i = a.level;
  const uint32_t lab = P.label[i];
  const uint32_t nc = P.ncons[i];
  uint32_t best;
  bs = 0;
  bci = DCI_BUCKET;
  ch = chc = 0;
  if (P.zero) {
    best = 0;
  } else if (nc == 0) {
    bs = __ldg(g.bucket_off + lab);
    best = __ldg(g.bucket_off + lab + 1) - bs;
    if (i == 0 && a.root_end) {
      const uint64_t rb = a.root_begin < best ? a.root_begin : uint64_t(best);
      const uint64_t re = a.root_end < best ? a.root_end : uint64_t(best);
      bs += uint32_t(rb);
      best = re > rb ? uint32_t((re - rb + a.root_step - 1) / a.root_step) : 0u;
    }
    ch = chc = (unsigned long long)best * (12ull + 4ull * g.W);
  } else {
    best = FULL;
    for (uint32_t c = 0; c < nc; ++c) {
      const uint32_t cs = P.cons[i][c];
      const uint32_t y = a.in.col[cs & 0xFF][r];
      uint32_t s, e;
      slice_of(g, cs >> 8, y, lab, s, e);
      ch += 8ull + 4ull * (e - s);
      if (e - s < best) {
        best = e - s;
        bs = s;
        bci = uint8_t(c);
      }
    }
    chc = (i + 1 == P.k && P.last_o1) ? 8ull : ch;
  }
  if (a.q_budget && best && a.in.qid) {
    // Per-query budget of a batch's rows (one query's are charged by the tile):
    // a query whose scheduled elements pass the budget stops expanding (its
    // count is reported as unknown).
    const unsigned long long before = atomicAdd(&a.q_elems[q], (unsigned long long)best);
    if (before + best > a.q_budget) best = 0;
  }
  return best;
}

__device__ __forceinline__ unsigned long long block_exclusive_scan(unsigned long long v,
                                                                   unsigned long long* total) {
  __shared__ unsigned long long wsum[33];
  const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  unsigned long long incl = v;
  for (int d = 1; d < 32; d <<= 1) {
    unsigned long long t = __shfl_up_sync(FULL, incl, d);
    if (lane >= d) incl += t;
  }
  if (lane == 31) wsum[wid] = incl;
  __syncthreads();
  if (wid == 0) {
    const uint32_t nw = blockDim.x >> 5;
    unsigned long long s = lane < nw ? wsum[lane] : 0ull;
    unsigned long long si = s;
    for (int d = 1; d < 32; d <<= 1) {
      unsigned long long t = __shfl_up_sync(FULL, si, d);
      if (lane >= d) si += t;
    }
    if (lane < nw) wsum[lane] = si - s;
    if (lane == nw - 1) wsum[32] = si;
  }
  __syncthreads();
  unsigned long long res = wsum[wid] + incl - v;
  *total = wsum[32];
  __syncthreads();
  return res;
}

// First row of every tile of the element range [t0, t1): tile_row[j] is the
// row holding element t0 + j*EXPAND_TILE (clamped to t1 - 1), j = 0..ntiles.
__global__ void __launch_bounds__(256) k_tile_rows(const uint64_t* __restrict__ woff, uint32_t R,
                                                   uint64_t t0, uint64_t t1, uint32_t ntiles,
                                                   uint32_t* tile_row) {
  for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j <= ntiles;
       j += gridDim.x * blockDim.x) {
    uint64_t t = t0 + uint64_t(j) * EXPAND_TILE;
    if (t > t1 - 1) t = t1 - 1;
    tile_row[j] = find_row(woff, 0, R - 1, t);
  }
}

// Launch shapes of the expand kernel, fixed at compile time so a launch
// carries only the code (and registers) of the paths its rows can take.
enum : int {
  X_WRITE = 1,  // survivors are appended to the next level table
  X_EMIT = 2,   // complete matches are written as rows (emit mode)
  X_FUSED = 4,  // the last position (one backward slice) is closed in place
  X_TAIL = 8,   // a two-position pendant tail is closed from dense aggregates
  X_ONE = 16,   // one query, no row query ids: its plan is staged in shared memory
  X_DIRECT = 32,  // with X_ONE and X_FUSED or X_TAIL: candidates are closed where they
                  // are found (see direct_sides)
  X_ALONE = 64,   // with X_DIRECT: the position has no further constraint
  X_PAIR = 128,   // with X_ONE: exactly one further constraint, at most two equal
                  // labels before, no self-loop, no matrix filter
  X_TRIO = 256,   // the same with two further constraints
};

// Positions of a row whose adjacency each candidate of position i is looked up
// in to be closed.  The slice that closes it (FUSED: of the last position, TAIL:
// of position k-2) is the candidate's own, and then earlier matches with that
// slice's label may lie in it, or that of an earlier vertex, and then the
// candidate itself may; what earlier matches take from it is a matter of the row.
__host__ __device__ __forceinline__ uint32_t direct_sides(const PlanDev& P, uint32_t i, bool tail) {
  const uint32_t anchor = tail ? P.tail_p : P.cons[P.k - 1][0] & 0xFF;
  const uint32_t open = tail ? P.tail_Ia : P.samelab[P.k - 1] & ~P.guar[P.k - 1];
  if (anchor == i) return open & ((1u << i) - 1);
  return (open >> i) & 1u ? 1u << anchor : 0u;
}

// One set-up row of an expand task (shared memory, a row per slot).  A further
// constraint is probed at p: the hub bitmap row of its vertex (len HUB_LEN), or
// its sorted label slice of len entries.  The stride of 80 bytes keeps 16-byte
// reads of eight consecutive rows free of bank conflicts.
struct alignas(16) XRow {
  const uint32_t* list;  // list[e] is element e of the task (nullptr: a bucket row)
  const uint32_t* p0;    // first further constraint
  uint32_t len0, m0;     // m0, m1: earlier matches a candidate must differ from
  uint32_t row, beg;     // table row; its first element of the task
  const uint32_t* p1;    // second further constraint
  uint32_t len1, m1;
  uint32_t q, ci, v0;    // query; driving constraint; bucket row: element e is
  uint32_t end;          // vertex v0 + e * root_step
  // X_DIRECT, slice of an earlier vertex: its entries, those that no earlier
  // match takes, and a tail's matches and second-slice entries over them.
  uint32_t raw, free, c0, d0;
};
constexpr uint32_t HUB_LEN = FULL;

// Probe data of constraint cs for row r (see XRow); an empty slice points at
// readable memory.
__device__ __forceinline__ void probe_of(const StepArgs& a, uint32_t cs, uint32_t lab, uint32_t r,
                                         const uint32_t*& p, uint32_t& len) {
  const GraphDev& g = a.g;
  const uint32_t d = cs >> 8;
  const uint32_t y = a.in.col[cs & 0xFF][r];
  uint32_t h = NO_HUB, s = 0, e = 0;
  if (g.hub_slot[d]) h = __ldg(g.hub_slot[d] + y);
  if (h == NO_HUB || a.probe_min > 1) slice_of(g, d, y, lab, s, e);
  if (h == NO_HUB || (a.probe_min > 1 && e - s < a.probe_min)) {
    p = e > s ? g.adj[d] + s : g.bucket_off;
    len = e - s;
  } else {
    p = g.hub_bits[d] + uint64_t(h) * g.hub_words;
    len = HUB_LEN;
  }
}

// Probes U candidates per lane, each against a constraint of its own: p[u],
// len[u] as in XRow; ok[u] is cleared where x[u] is not in it.  No load hangs
// on a condition, so the loads of the U candidates overlap.  Searches halve
// together until the longest slice of the warp is done.
template <int U>
__device__ __forceinline__ void probe_all(const uint32_t* const (&p)[U], const uint32_t (&len)[U],
                                          const uint32_t (&x)[U], bool (&ok)[U]) {
  uint32_t w[U], longest = 0;
#pragma unroll
  for (int u = 0; u < U; ++u) {
    w[u] = __ldg(p[u] + (len[u] == HUB_LEN ? x[u] >> 5 : 0u));
    ok[u] = ok[u] && len[u];  // nothing lies in an empty slice
    if (len[u] != HUB_LEN && ok[u]) longest = max(longest, len[u]);
  }
  longest = __reduce_max_sync(FULL, longest);
  if (longest) {
    uint32_t at[U], n[U];  // the last entry <= x[u], if any, lies in [at, at + n)
#pragma unroll
    for (int u = 0; u < U; ++u) {
      at[u] = 0;
      n[u] = len[u] == HUB_LEN ? 0u : len[u];
    }
    for (; longest > 1; longest -= longest >> 1) {
      uint32_t v[U];
#pragma unroll
      for (int u = 0; u < U; ++u) v[u] = __ldg(p[u] + (at[u] + (n[u] >> 1)));
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const uint32_t half = n[u] >> 1;
        at[u] += v[u] <= x[u] ? half : 0u;
        n[u] -= half;
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint32_t v = __ldg(p[u] + at[u]);
      if (len[u] != HUB_LEN) ok[u] = ok[u] && v == x[u];
    }
  }
#pragma unroll
  for (int u = 0; u < U; ++u)
    if (len[u] == HUB_LEN) ok[u] = ok[u] && ((w[u] >> (x[u] & 31)) & 1u);
}

// Expand kernel: a warp takes tasks of up to EXPAND_TILE consecutive elements
// (row, driving entry).
//
// What bounds it: chains of dependent loads that mostly hit L2 (row offset ->
// matched vertices -> hub slot or slice -> candidate -> probe), and then the
// instructions per candidate.  So
//   * the state of a row (XRow) is set up for 32 rows at once, a row per lane,
//     and kept in shared memory: one chain of loads per 32 rows;
//   * candidates are taken 32 * XU at a time whatever their rows, every lane
//     finding its rows by the row starts up to its element; the candidates of
//     the next group are loaded while this one is probed, and the XU probes of
//     a lane are independent loads;
//   * survivors are staged in shared memory, so that what follows them
//     (filters, closed forms, appending to the next table, emitting) runs on
//     full warps, with one reservation per staged group and no block barriers.
// Against one element per thread with a search for its row in global memory
// and 256-thread tiles (R-MAT scale 22): 4-cycle 15.7 -> 11.9 ms, 4-clique
// 12.1 -> 7.3 ms, 256 batched queries 110 -> 67 ms.  A table that overflows is
// flagged once per warp, not once per survivor: runs past their budget on
// scale 20 took 577 ms and take 65.  Two candidates a lane (XU) and four
// blocks per SM (64 registers) were the best of 1-4 and 3-6: more candidates
// spill, fewer expose the probe latency.  Walking each row by its own, 32-128
// candidates at a time, was no better (11.3-12.5 ms for the 4-cycle).
//
// X_DIRECT leaves the staging out where nearly every candidate survives and is
// closed at once, with its look-ups done like the probes of the others:
// instructions per candidate were what bounded those launches (275 per 32
// candidates, 71% issue).  R-MAT scale 18, 5-paths whose ends share a label:
// 90 -> 184 and 47 -> 191 G candidates/s; scale 22, 5-path: 6.5 -> 5.5 ms, and
// 2.6 ms with all a tail needs in one 16-byte table entry instead of six loads
// (3.6 ms at four blocks per SM with 64 registers; the tail shapes get three blocks
// and 80 registers, of which 56 and 120 still spill 36 and 44 bytes and 24 spills 24).
//
// X_PAIR, the commonest shape (two lists intersected), leaves out what the
// others may need and has the registers for three candidates a lane: 4-cycle
// 8.9 -> 7.9 ms, triangle 1.62 -> 1.40 ms on scale 22 (two candidates 8.3 ms,
// four 8.5; five blocks per SM 9.2, three 8.6-8.9).  X_TRIO is the same for three
// lists: 4-cliques of six labellings on scale 22, 4.57 -> 4.35 ms a call (three
// candidates 4.39).
template <int MODE>
__global__ void __launch_bounds__(EXPAND_BLOCK, (MODE & X_TAIL) ? 3 : 4) k_expand(StepArgs a) {
  constexpr bool ONE = (MODE & X_ONE) != 0;
  // Launches that only count complete matches keep nothing of a survivor.
  constexpr bool DIRECT = (MODE & X_DIRECT) != 0;
  constexpr bool STAGE = ((MODE & (X_WRITE | X_EMIT | X_FUSED | X_TAIL)) != 0 || !ONE) && !DIRECT;
  constexpr int XU = (MODE & X_PAIR) ? 3 : 2;
  const uint32_t i = a.level;
  const GraphDev& g = a.g;
  const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  __shared__ XRow s_rows[EXPAND_BLOCK / 32][32];
  __shared__ uint32_t s_x[STAGE ? EXPAND_BLOCK / 32 : 1][STAGE ? XSTAGE : 1];
  __shared__ uint32_t s_r[STAGE ? EXPAND_BLOCK / 32 : 1][STAGE ? XSTAGE : 1];
  // A single query's plan is read by every row: staged once per block.
  __shared__ PlanDev s_plan;
  chain_begin();
  if constexpr (ONE) {
    const uint32_t* src = reinterpret_cast<const uint32_t*>(a.plans);
    uint32_t* dst = reinterpret_cast<uint32_t*>(&s_plan);
    for (uint32_t w = threadIdx.x; w < sizeof(PlanDev) / 4; w += EXPAND_BLOCK) dst[w] = src[w];
    __syncthreads();
  }
  chain_wait();
  uint64_t t0 = a.t0, t1 = a.t1;
  if (a.dev) {
    // (a lane whose tables overflowed stops: its query is counted again)
    t0 = 0;
    t1 = ONE && i == 0 ? a.T0 : a.ctr[lvl_slot(int(i), L_T)];
    // Other warps of this launch may set C_ERR meanwhile: a warp leaves as a
    // whole, on what its first lane saw, and no block barrier follows.  C_STOP
    // and the sizes are left by kernels that have ended.
    const bool stopped = a.ctr[C_STOP] || (a.lane && __ldcg(&a.ctr[C_ERR])) || t1 > a.seg_cap;
    if (__shfl_sync(FULL, stopped ? 1 : 0, 0)) return;
  }
  const uint64_t span = t1 - t0;
  const uint32_t ntiles = uint32_t((span + EXPAND_TILE - 1) / EXPAND_TILE);
  auto plan = [&](uint32_t q) -> const PlanDev& { return ONE ? s_plan : a.plans[q]; };
  auto query = [&](uint32_t r) -> uint32_t { return !ONE && a.in.qid ? a.in.qid[r] : 0u; };
  // What candidates of this level are checked for (one query; a batch looks at
  // every row's plan): further constraints, equal labels, and the rare checks.
  constexpr bool ALONE = (MODE & X_ALONE) != 0;
  constexpr bool PAIR = (MODE & X_PAIR) != 0, TRIO = (MODE & X_TRIO) != 0;
  const uint32_t others = ALONE  ? 0u
                          : PAIR ? 1u
                          : TRIO ? 2u
                          : ONE  ? plan(0).ncons[i] - (plan(0).ncons[i] ? 1u : 0u)
                                 : 3u;
  const uint32_t sames = ONE ? __popc(plan(0).samelab[i]) : 3u;
  const bool extra =
      PAIR || TRIO ? false : (i == 0 && a.root_keep) || ((plan(0).selfloop_mask >> i) & 1u);

  // X_DIRECT: the vertices of a row that candidates are looked up in, in the
  // slots that further constraints leave.
  const uint32_t sides = DIRECT ? direct_sides(plan(0), i, (MODE & X_TAIL) != 0) : 0u;
  const uint32_t nsides = __popc(sides);
  const uint32_t kl = plan(0).k - 1;
  const uint32_t anchor = (MODE & X_TAIL) ? plan(0).tail_p : plan(0).cons[kl][0] & 0xFF;
  const bool own = anchor == i;  // the closing slice is the candidate's
  unsigned long long d_c = 0, d_raw = 0, d_d = 0;      // sums over closed candidates
  uint32_t d_in = 0;

  unsigned long long cnt = 0, bal = 0, balc = 0, s1 = 0, sk = 0, s2 = 0;
  uint32_t cnt_q = 0;
  bool full = false;  // the output table is full (lane pipeline)
  uint32_t staged = 0;

  // What follows the staged survivors.
  auto flush = [&]() {
    __syncwarp();
    uint32_t kept = 0;
    for (uint32_t v0 = 0; v0 < staged; v0 += 32) {
      bool ok = v0 + lane < staged;
      const uint32_t x = ok ? s_x[wid][v0 + lane] : 0u, rr = ok ? s_r[wid][v0 + lane] : 0u;
      const uint32_t q = ok ? query(rr) : 0u;
      const PlanDev& P = plan(q);
      const bool fin = i + 1 == P.k;
      bool fused = false, ftail = false;
      if constexpr ((MODE & X_FUSED) != 0)
        fused = !fin && a.count_mode && (i + 2 == P.k) && P.last_o1;
      if constexpr ((MODE & X_TAIL) != 0)
        ftail = ((a.tail_dense && P.tail2) || (a.star && P.star2)) && i + 3 == P.k;
      // Filters prune positions whose survivors are extended further; the
      // position before a last position counted in closed form is not
      // filtered (the closed form already yields 0 for hopeless candidates).
      if (ok && !fin && a.filters && !(i + 2 == P.k && P.last_o1))
        ok = pass_filters(g, P, i, x, a.filters);
      if (ok) {
        if constexpr (!ONE) {
          if (q != cnt_q) {
            acc_flush(a, cnt_q, i, cnt, s1, sk, s2);
            cnt = s1 = sk = s2 = 0;
            cnt_q = q;
          }
        }
        s1 += 1;
        if (fin) {
          if (!ONE && a.count_mode) cnt += 1;
        } else if ((MODE & X_TAIL) && ftail && P.star2) {
          // The prefix ending in x has length k-2 and the plan ends in two
          // leaves of one anchor: counted here, not stored.
          unsigned long long tc, tp, tb, tbc;
          star_close(a, P, [&](uint32_t j) { return j == i ? x : a.in.col[j][rr]; },
                     P.star_p == i, tc, tp, tb, tbc);
          cnt += tc;
          sk += tc;
          s2 += tp;
          bal += tb;
          balc += tbc;
        } else if ((MODE & X_TAIL) && ftail) {
          // The prefix ending in x has length k-2: its two-position pendant
          // tail is counted here from the dense aggregates, not stored.
          const uint32_t mp = P.tail_p == i ? x : a.in.col[P.tail_p][rr];
          const uint4 te = tail_entry(a, P, mp);
          unsigned long long tc, tp, td;
          tail_close(a, P, [&](uint32_t j) { return j == i ? x : a.in.col[j][rr]; }, P.tail_Ia, mp,
                     P.tail_p == i, te, tc, tp, td);
          cnt += tc;
          sk += tc;
          s2 += tp;
          bal += 8ull + 4ull * te.z + 8ull * tp + 4ull * td;
          balc += 8ull + 4ull * te.z + 8ull * tp;
        } else if ((MODE & X_FUSED) && fused) {
          const uint32_t kl = P.k - 1;
          const uint32_t cs = P.cons[kl][0];
          const uint32_t pos = cs & 0xFF, dir = cs >> 8;
          const uint32_t y = pos == i ? x : a.in.col[pos][rr];
          uint32_t s, en;
          slice_of(g, dir, y, P.label[kl], s, en);
          uint32_t c1 = en - s;
          bal += 8ull + 4ull * c1;
          balc += 8ull;
          for (uint32_t m = P.samelab[kl]; m; m &= m - 1) {
            const uint32_t j = __ffs(m) - 1;
            if ((P.guar[kl] >> j) & 1u) {
              c1 -= 1;
            } else {
              const uint32_t mj = j == i ? x : a.in.col[j][rr];
              c1 -= joined(a, dir, y, P.label[pos], pos == i, s, en, mj) ? 1u : 0u;
            }
          }
          sk += c1;
          cnt += c1;
        }
      }
      if constexpr ((MODE & (X_WRITE | X_EMIT)) != 0) {
        // compact what stays, in place
        const bool keep = ok && !fused && !ftail && fin == ((MODE & X_EMIT) != 0);
        const uint32_t km = __ballot_sync(FULL, keep);
        if (keep) {
          const uint32_t at = kept + __popc(km & lanemask_lt());
          s_x[wid][at] = x;
          s_r[wid][at] = rr;
        }
        kept += __popc(km);
      } else if (ok && !fin && !fused && !ftail) {  // no table to append to
        atomicOr(&a.ctr[C_ERR], (unsigned long long)ERR_OVERFLOW);
      }
    }
    if constexpr ((MODE & (X_WRITE | X_EMIT)) != 0) {
      __syncwarp();
      if (kept) {
        const uint32_t slot = (MODE & X_EMIT) ? uint32_t(C_EMIT) : a.out_slot;
        const uint64_t cap = (MODE & X_EMIT) ? a.emit_cap : a.out_cap;
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd(&a.ctr[slot], (unsigned long long)kept);
        base = __shfl_sync(FULL, base, 0);
        if (base + kept > cap) {
          // flagged once per warp; nothing is written past the table
          if (lane == 0) atomicOr(&a.ctr[C_ERR], (unsigned long long)ERR_OVERFLOW);
          full = true;
          kept = base < cap ? uint32_t(cap - base) : 0u;
        }
        if constexpr ((MODE & X_EMIT) != 0) {
          for (uint32_t v = lane; v < kept; v += 32) {
            const uint32_t rr = s_r[wid][v];
            unsigned long long key = 0;
            for (uint32_t j = 0; j <= i; ++j) {
              const uint32_t y = j < i ? a.in.col[j][rr] : s_x[wid][v], u = s_plan.perm[j];
              const uint32_t id = __ldg(g.globalid + y);
              if (a.emit_key)
                key |= (unsigned long long)id << ((a.emit_k - 1 - u) * a.emit_bits);
              else
                a.emit_col[u][base + v] = id;
            }
            if (a.emit_key) a.emit_key[base + v] = key;
          }
        } else {
          for (uint32_t v = lane; v < kept; v += 32) {
            const uint32_t rr = s_r[wid][v];
            for (uint32_t j = 0; j < i; ++j) a.out.col[j][base + v] = a.in.col[j][rr];
            a.out.col[i][base + v] = s_x[wid][v];
            if (!ONE && a.out.qid) a.out.qid[base + v] = query(rr);
          }
        }
      }
    }
    __syncwarp();  // the stage is filled again
    staged = 0;
  };

  // A launch with fewer tiles than warps splits its tiles into parts of down
  // to 64 elements, so that small levels still use every warp; a large one
  // takes several tiles per grab of the work queue.  The first grab is by warp
  // index, the queue serves the others.
  const uint32_t nwarps = gridDim.x * (EXPAND_BLOCK / 32);
  uint32_t split = 0;  // parts per tile, as a power of two
  while ((EXPAND_TILE >> split) > 64 && (ntiles << (split + 1)) <= nwarps) ++split;
  const uint32_t ntasks = ntiles << split;
  const uint32_t part = EXPAND_TILE >> split;
  uint32_t grab = a.grab;
  if (!grab) {
    grab = ntasks / (nwarps * 8);
    grab = grab < 1 ? 1 : (grab > 16 ? 16 : grab);
  }
  const uint32_t rstep = i == 0 ? a.root_step : 1u;  // stride of the level-0 candidates
  const bool root = ONE && i == 0;                   // one row, no table
  XRow* rows = s_rows[wid];
  uint64_t gbase = uint64_t(blockIdx.x * (EXPAND_BLOCK / 32) + wid) * grab;
  while (gbase < ntasks && !full) {
    const uint32_t gend = uint32_t(min(gbase + grab, uint64_t(ntasks)));
    for (uint32_t task = uint32_t(gbase); task < gend && !full; ++task) {
      const uint32_t tile = task >> split;
      uint64_t t = t0 + uint64_t(tile) * EXPAND_TILE + (task & ((1u << split) - 1)) * part;
      const uint64_t te = min(t + part, t1);
      if (t >= te) continue;
      uint32_t r0 = root ? 0u : a.tile_row[tile];
      const uint32_t rhi = root ? 0u : a.tile_row[tile + 1];
      while (t < te && !full) {
        if (r0 < rhi) r0 = find_row(a.woff, r0, rhi, t);
        // Set up 32 rows, one per lane: consecutive ones, or, where more rows
        // than elements are left (many are empty), the rows of the next 32
        // elements.
        const uint32_t left = uint32_t(te - t);
        uint32_t row = min(r0 + lane, rhi);
        bool mine = r0 + lane <= rhi;
        if (rhi - r0 >= 32 && rhi - r0 > left) {
          row = find_row(a.woff, r0, rhi, min(t + lane, te - 1));
          const uint32_t prev = __shfl_up_sync(FULL, row, 1);
          mine = lane == 0 || row != prev;
        }
        const uint64_t o0 = root ? 0ull : a.woff[row], o1 = root ? a.T0 : a.woff[row + 1];
        // the row's elements in this task, relative to t
        const uint32_t beg = uint32_t(min(max(o0, t), te) - t);
        const uint32_t end = uint32_t(min(max(o1, t), te) - t);
        mine = mine && end > beg;
        const uint32_t act = __ballot_sync(FULL, mine);
        const uint32_t nrows = __popc(act);
        __syncwarp();  // the previous rows are no longer read
        if (mine) {
          XRow R;
          R.row = row;
          R.q = query(row);
          R.beg = beg;
          R.end = end;
          const PlanDev& P = plan(R.q);
          const uint32_t lab = P.label[i], nc = P.ncons[i];
          const uint32_t ci = root ? uint32_t(DCI_BUCKET) : uint32_t(a.dci[row]);
          const uint32_t ds = root ? a.root_first : a.dstart[row];
          const uint64_t skip = t + beg - o0;  // elements of the row before the task
          R.list = ci == DCI_BUCKET ? nullptr
                                    : g.adj[P.cons[i][ci] >> 8] + int64_t(ds + skip) - beg;
          R.v0 = ds + uint32_t(skip) * rstep - beg * rstep;
          R.ci = ci;
          R.m0 = R.m1 = FULL;
          uint32_t m = P.samelab[i];
          if (m) {
            R.m0 = a.in.col[__ffs(m) - 1][row];
            m &= m - 1;
            if (m) R.m1 = a.in.col[__ffs(m) - 1][row];
          }
          R.p0 = R.p1 = nullptr;
          R.len0 = R.len1 = 0;
          uint32_t c = ci == 0 ? 1u : 0u;
          if (c < nc) {
            probe_of(a, P.cons[i][c], lab, row, R.p0, R.len0);
            if (++c == ci) ++c;
            if (!PAIR && c < nc) probe_of(a, P.cons[i][c], lab, row, R.p1, R.len1);
          }
          if constexpr (DIRECT) {
            uint32_t slot = others;
            for (uint32_t m2 = sides; m2; m2 &= m2 - 1, ++slot)
              probe_of(a, __ffs(m2) - 1, lab, row, slot ? R.p1 : R.p0, slot ? R.len1 : R.len0);
            if (!own) {
              const uint32_t y = a.in.col[anchor][row];
              if constexpr ((MODE & X_TAIL) != 0) {
                const uint4 te = tail_entry(a, P, y);
                unsigned long long tc, tp, td;
                tail_close(a, P, [&](uint32_t j) { return a.in.col[j][row]; },
                           P.tail_Ia & ((1u << i) - 1), y, false, te, tc, tp, td);
                R.raw = te.z;
                R.free = uint32_t(tp);
                R.c0 = uint32_t(tc);
                R.d0 = uint32_t(td);
              } else {
                uint32_t s, e;
                slice_of(g, P.cons[kl][0] >> 8, y, P.label[kl], s, e);
                R.raw = R.free = e - s;
                for (uint32_t m2 = P.samelab[kl] & ((1u << i) - 1); m2; m2 &= m2 - 1) {
                  const uint32_t j = __ffs(m2) - 1;
                  R.free -= ((P.guar[kl] >> j) & 1u) ||
                            in_slice_se(g, P.cons[kl][0] >> 8, y, s, e, a.in.col[j][row],
                                        a.probe_min);
                }
              }
            }
          }
          rows[__popc(act & lanemask_lt())] = R;
        }
        __syncwarp();
        const uint32_t covered = rows[nrows - 1].end;  // elements these rows hold
        const uint32_t mybeg = lane < nrows ? rows[lane].beg : FULL;
        uint32_t before = 0;  // rows that begin before the next group
        uint32_t x[XU], h[XU], xn[XU], hn[XU];
        // Candidates and row slots of the elements from e0 on (past the last
        // element: the last element's).
        auto load = [&](uint32_t e0, uint32_t (&xx)[XU], uint32_t (&hh)[XU]) {
#pragma unroll
          for (int u = 0; u < XU; ++u) {
            const uint32_t d = mybeg - (e0 + u * 32);
            const uint32_t starts = __reduce_or_sync(FULL, d < 32 ? 1u << d : 0u);
            hh[u] = before + __popc(starts & (lanemask_lt() | (1u << lane))) - 1;
            before += __popc(starts);
          }
#pragma unroll
          for (int u = 0; u < XU; ++u) {
            const uint32_t e = min(e0 + u * 32 + lane, covered - 1);
            const XRow& R = rows[hh[u]];
            if (R.list) xx[u] = __ldg(R.list + e);
            else xx[u] = R.v0 + e * rstep;
          }
        };
        load(0, xn, hn);
        for (uint32_t e0 = 0; e0 < covered && !full; e0 += 32 * XU) {
          bool ok[XU];
#pragma unroll
          for (int u = 0; u < XU; ++u) {
            x[u] = xn[u];
            h[u] = hn[u];
            ok[u] = e0 + u * 32 + lane < covered;
          }
          if (e0 + 32 * XU < covered) load(e0 + 32 * XU, xn, hn);
          // (in a batch a row may have no such constraint)
          auto probe_some = [&](const uint32_t* (&p)[XU], uint32_t (&len)[XU]) {
            if constexpr (ONE) {
              probe_all<XU>(p, len, x, ok);
            } else {
              bool in[XU];
#pragma unroll
              for (int u = 0; u < XU; ++u) {
                in[u] = ok[u] && p[u];
                if (!p[u]) p[u] = g.bucket_off;
              }
              bool res[XU];
#pragma unroll
              for (int u = 0; u < XU; ++u) res[u] = in[u];
              probe_all<XU>(p, len, x, res);
#pragma unroll
              for (int u = 0; u < XU; ++u) ok[u] = in[u] ? res[u] : ok[u];
            }
          };
          if (sames || !ONE) {
#pragma unroll
            for (int u = 0; u < XU; ++u)
              ok[u] = ok[u] && x[u] != rows[h[u]].m0 && x[u] != rows[h[u]].m1;
          }
          if (others > 0 || !ONE) {
            const uint32_t* p[XU];
            uint32_t len[XU];
#pragma unroll
            for (int u = 0; u < XU; ++u) {
              p[u] = rows[h[u]].p0;
              len[u] = rows[h[u]].len0;
            }
            probe_some(p, len);
          }
          if (others > 1 || !ONE) {
            const uint32_t* p[XU];
            uint32_t len[XU];
#pragma unroll
            for (int u = 0; u < XU; ++u) {
              p[u] = rows[h[u]].p1;
              len[u] = rows[h[u]].len1;
            }
            probe_some(p, len);
          }
          // constraints and equal labels past the two that a row keeps, and the
          // rare checks
          if (!PAIR && !TRIO && (others > 2 || sames > 2 || extra)) {
#pragma unroll
            for (int u = 0; u < XU; ++u) {
              if (!ok[u]) continue;
              const XRow& R = rows[h[u]];
              const PlanDev& P = plan(R.q);
              uint32_t m = P.samelab[i];
              m &= m - 1;
              for (m &= m - 1; m && ok[u]; m &= m - 1)
                ok[u] = a.in.col[__ffs(m) - 1][R.row] != x[u];
              const uint32_t k0 = R.ci == 0 ? 1u : 0u, k1 = k0 + 1 == R.ci ? k0 + 2 : k0 + 1;
              for (uint32_t c = k1 + 1; c < P.ncons[i] && ok[u]; ++c) {
                if (c == R.ci) continue;
                const uint32_t cs = P.cons[i][c];
                ok[u] = in_slice(g, cs >> 8, a.in.col[cs & 0xFF][R.row], P.label[i], x[u],
                                 a.probe_min);
              }
              // the lossy matrix filter drops level-0 candidates it rejects
              if (i == 0 && a.root_keep && ok[u])
                ok[u] = (__ldg(a.root_keep + (x[u] >> 5)) >> (x[u] & 31)) & 1u;
              if (ok[u] && ((P.selfloop_mask >> i) & 1u)) ok[u] = has_self(g, x[u]);
            }
          }
          if constexpr (DIRECT) {
            // membership of the candidate in the sides' adjacency
            bool in0[XU], in1[XU];
#pragma unroll
            for (int u = 0; u < XU; ++u) in0[u] = in1[u] = false;
            auto look = [&](bool second, bool (&in)[XU]) {
              const uint32_t* p[XU];
              uint32_t len[XU];
#pragma unroll
              for (int u = 0; u < XU; ++u) {
                p[u] = second ? rows[h[u]].p1 : rows[h[u]].p0;
                len[u] = second ? rows[h[u]].len1 : rows[h[u]].len0;
                in[u] = ok[u];
              }
              probe_all<XU>(p, len, x, in);
            };
            if (nsides > 0) look(others > 0, in0);
            if (nsides > 1) look(true, in1);
            const PlanDev& P = s_plan;
            if constexpr ((MODE & X_FUSED) != 0) {
              const uint32_t* off = g.loff[P.cons[kl][0] >> 8] + uint64_t(P.label[kl]) * g.n;
              const uint32_t sure = __popc(P.samelab[kl] & P.guar[kl]);
              const bool self = own && ((P.samelab[kl] & ~P.guar[kl]) >> i & 1u);
              uint32_t raw[XU], free[XU];
#pragma unroll
              for (int u = 0; u < XU; ++u) {
                raw[u] = free[u] = 0;
                if (own) {
                  if (others == 0 || ok[u]) raw[u] = __ldg(off + x[u] + 1) - __ldg(off + x[u]);
                  free[u] = raw[u] - sure;
                } else {
                  raw[u] = rows[h[u]].raw;
                  free[u] = rows[h[u]].free - ((P.samelab[kl] & P.guar[kl]) >> i & 1u);
                }
              }
#pragma unroll
              for (int u = 0; u < XU; ++u)
                if (ok[u]) {
                  s1 += 1;
                  d_raw += raw[u];
                  d_c += free[u] - (in0[u] ? 1u : 0u) - (in1[u] ? 1u : 0u) -
                         (self && has_self(g, x[u]) ? 1u : 0u);
                }
            } else {
              // The filter of position i: its query neighbours are its backward
              // ones, which satisfy it by themselves, and, when the tail hangs
              // off the candidate, position k-2: its label is met when that
              // slice has entries.
              const uint32_t nJ = __popc(P.tail_J);
              const uint32_t min_len = own && (a.filters & MG_FILTER_NLB) ? 1u : 0u;
              const uint32_t min_deg = own && (a.filters & MG_FILTER_DEGREE) ? P.req[0][i] : 0u;
              const bool self = own && (P.tail_Ia >> i & 1u);
              uint4 te[XU];
              if (own) {
#pragma unroll
                for (int u = 0; u < XU; ++u) {
                  te[u] = make_uint4(0, 0, 0, 0);
                  if (others == 0 || ok[u]) te[u] = tail_entry(a, P, x[u]);
                }
              }
#pragma unroll
              for (int u = 0; u < XU; ++u) {
                if (!ok[u] || (own && (te[u].z < min_len || te[u].w < min_deg))) continue;
                const XRow& R = rows[h[u]];
                s1 += 1;
                if (in0[u] || in1[u] || (self && has_self(g, x[u]))) {
                  const uint32_t mp = own ? x[u] : a.in.col[anchor][R.row];
                  const uint4 t4 = own ? te[u] : tail_entry(a, P, mp);
                  unsigned long long tc, tp, td;
                  tail_close(a, P, [&](uint32_t j) { return j == i ? x[u] : a.in.col[j][R.row]; },
                             P.tail_Ia, mp, own, t4, tc, tp, td);
                  d_raw += t4.z;
                  d_c += tc;
                  d_d += td;
                  d_in += t4.z - uint32_t(tp);
                } else if (own) {
                  d_raw += te[u].z;
                  d_c += (unsigned long long)((long long)te[u].x - (long long)nJ * te[u].z);
                  d_d += te[u].y;
                } else {
                  d_raw += R.raw;
                  d_c += R.c0;
                  d_d += R.d0;
                  d_in += R.raw - R.free;
                }
              }
            }
          } else if constexpr (STAGE) {
#pragma unroll
            for (int u = 0; u < XU; ++u) {
              const uint32_t km = __ballot_sync(FULL, ok[u]);
              if (ok[u]) {
                const uint32_t w = staged + __popc(km & lanemask_lt());
                s_x[wid][w] = x[u];
                s_r[wid][w] = rows[h[u]].row;
              }
              staged += __popc(km);
            }
            // a task's survivors stay contiguous in the output
            if (staged > XSTAGE - 32 * XU ||
                (staged && e0 + 32 * XU >= covered && t + covered >= te))
              flush();
          } else {
            uint32_t n = 0;
#pragma unroll
            for (int u = 0; u < XU; ++u) n += ok[u] ? 1u : 0u;
            s1 += n;
          }
        }
        t += covered;
        if (r0 + 32 <= rhi && t < te) r0 = __shfl_sync(FULL, row, 31);
      }
      // In a batch: fold the per-thread counts of a warp that holds one query.
      if (!ONE && a.in.qid) acc_flush_warp(a, cnt_q, i, cnt, s1, sk, s2, false);
    }
    if (uint64_t(nwarps) * grab >= ntasks) break;  // the first grabs were all
    if (lane == 0) gbase = atomicAdd(&a.ctr[a.tile_slot], (unsigned long long)grab);
    gbase = __shfl_sync(FULL, gbase, 0) + uint64_t(nwarps) * grab;
  }
  if (ONE && a.count_mode && s_plan.k == i + 1) cnt = s1;  // complete matches
  if constexpr (DIRECT) {
    cnt = sk = d_c;
    if constexpr ((MODE & X_TAIL) != 0) {
      s2 = d_raw - d_in;
      balc = 8 * s1 + 4 * d_raw + 8 * s2;
      bal = balc + 4 * d_d;
    } else {
      balc = 8 * s1;
      bal = 8 * s1 + 4 * d_raw;
    }
  }
  acc_flush_warp(a, cnt_q, i, cnt, s1, sk, s2, true);
  bal = warp_sum(bal);
  balc = warp_sum(balc);
  if (lane == 0 && (bal | balc)) {
    atomicAdd(&a.ctr[C_BALG], bal);
    atomicAdd(&a.ctr[C_BALGC], balc);
  }
}

// ---- work and scan -----------------------------------------------------------
// Sum of the tiles before `tile` (decoupled look-back by one warp, 32
// predecessors at a time: back to the nearest inclusive prefix).  A tile only
// waits for tiles claimed before it, whose blocks are running; every wait gives
// up after spin_limit polls (ERR_TIMEOUT).
__device__ __forceinline__ unsigned long long look_back(const StepArgs& a, uint32_t epoch,
                                                        uint64_t tile) {
  const uint32_t lane = threadIdx.x & 31;
  unsigned long long prefix = 0;
  for (int64_t t = int64_t(tile) - 1; t >= 0; t -= 32) {
    const int64_t at = t - int64_t(lane);
    unsigned long long w = lb_word(epoch, LB_INC, 0);  // before the first tile
    if (at >= 0) {
      volatile unsigned long long* st = a.scan_status + at;
      uint32_t spins = 0;
      for (;;) {
        w = *st;
        if (lb_epoch(w) == epoch && lb_state(w)) break;
        if (++spins > a.spin_limit) {
          atomicOr(&a.ctr[C_ERR], (unsigned long long)ERR_TIMEOUT);
          w = lb_word(epoch, LB_INC, 0);
          break;
        }
        __nanosleep(32);
      }
    }
    __syncwarp();
    const uint32_t inc = __ballot_sync(FULL, lb_state(w) == LB_INC);
    const uint32_t upto = inc ? __ffs(inc) - 1 : 31u;
    unsigned long long v = lane <= upto ? lb_value(w) : 0ull;
    v = warp_sum(v);
    prefix += __shfl_sync(FULL, v, 0);
    if (inc) break;
  }
  return prefix;
}

// Work and scan of one level in one pass: tiles of WS_ROWS rows are taken in
// launch order from a counter; each computes its rows' driving slices (the
// shortest backward slice, or the label bucket for a position without backward
// neighbours) and their algorithmic-byte charge, publishes its sum, adds the
// sums of the tiles before it, and writes its rows' element offsets and the
// first row of every expand tile that begins among its elements.  The last
// tile writes the level's element total; a total past t_limit (or, on a lane,
// past seg_cap) stops the walk before the level is expanded.
//
// One launch and one pass over the rows in place of a work kernel, three scan
// kernels and a tile-row search, with no size returned to the host.  Five blocks
// per SM (48 registers) is what the compiler takes by itself, but unasked it
// spills 28 bytes there.
__global__ void __launch_bounds__(256, 5) k_work_scan(StepArgs a, uint32_t epoch) {
  const uint32_t i = a.level;
  chain_begin();
  chain_wait();
  const uint64_t R = dev_rows(a);
  const uint64_t ntiles = (R + WS_ROWS - 1) / WS_ROWS;
  unsigned long long bal = 0, balc = 0;
  __shared__ uint32_t s_tile;
  __shared__ unsigned long long s_prefix;
  __shared__ unsigned long long s_off[WS_ROWS];
  const PlanDev& P0 = a.plans[0];
  const uint32_t nc = P0.ncons[i];
  const bool o1 = i + 1 == P0.k && P0.last_o1;
  const bool fast = !a.in.qid && i > 0 && nc > 0 && !P0.zero;
  for (;;) {
    // One thread looks at the flags, because this launch sets them too (the last
    // tile's block C_STOP, any block C_ERR) while blocks without a tile are still
    // starting: a block leaves or stays as a whole.
    if (threadIdx.x == 0) {
      const uint64_t claimed = atomicAdd(&a.ctr[lvl_slot(int(i), L_SCAN)], 1ull);
      const bool stopped = __ldcg(&a.ctr[C_STOP]) || __ldcg(&a.ctr[C_ERR]);
      s_tile = stopped || claimed >= ntiles ? FULL : uint32_t(claimed);
    }
    __syncthreads();
    const uint32_t tile = s_tile;
    __syncthreads();
    if (tile == FULL) break;
    const uint64_t base = uint64_t(tile) * WS_ROWS + uint64_t(threadIdx.x) * 4;
    unsigned long long v[4] = {}, sum = 0;
    if (fast && base + 4 <= R) {
      // Four rows of one query at once: their columns are one 16-byte read, and
      // the reads of their slices overlap.
      uint32_t best[4], bs[4], ci[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        best[j] = FULL;
        bs[j] = ci[j] = 0;
      }
      unsigned long long ch = 0;
      const uint32_t lab = P0.label[i];
      for (uint32_t c = 0; c < nc; ++c) {
        const uint32_t cs = P0.cons[i][c];
        const uint4 y4 = *reinterpret_cast<const uint4*>(a.in.col[cs & 0xFF] + base);
        const uint32_t y[4] = {y4.x, y4.y, y4.z, y4.w};
        uint32_t s[4], e[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) slice_of(a.g, cs >> 8, y[j], lab, s[j], e[j]);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          ch += e[j] - s[j];
          if (e[j] - s[j] < best[j]) {
            best[j] = e[j] - s[j];
            bs[j] = s[j];
            ci[j] = c;
          }
        }
      }
      bal += 32ull * nc + 4 * ch;
      balc += o1 ? 32ull : 32ull * nc + 4 * ch;
      *reinterpret_cast<uint4*>(a.dstart + base) = make_uint4(bs[0], bs[1], bs[2], bs[3]);
      *reinterpret_cast<uchar4*>(a.dci + base) = make_uchar4(ci[0], ci[1], ci[2], ci[3]);
#pragma unroll
      for (int j = 0; j < 4; ++j) sum += v[j] = best[j];
    } else {
      for (int j = 0; j < 4; ++j) {
        const uint64_t r = base + j;
        if (r >= R) break;
        const uint32_t q = a.in.qid ? a.in.qid[r] : 0u;
        uint32_t bs;
        uint8_t bci;
        unsigned long long ch, chc;
        v[j] = row_work(a, a.plans[q], r, q, bs, bci, ch, chc);
        a.dstart[r] = bs;
        a.dci[r] = bci;
        bal += ch;
        balc += chc;
        sum += v[j];
      }
    }
    unsigned long long tot;
    unsigned long long ex = block_exclusive_scan(sum, &tot);
    if (a.q_budget && !a.in.qid) {
      // One query: a tile whose elements pass its budget is not expanded (the
      // count is reported as unknown).
      if (threadIdx.x == 0) s_prefix = atomicAdd(&a.q_elems[0], tot);
      __syncthreads();
      if (s_prefix + tot > a.q_budget) {
        tot = ex = 0;
        for (int j = 0; j < 4; ++j) v[j] = 0;
      }
      __syncthreads();
    }
    if (threadIdx.x < 32) {
      if (threadIdx.x == 0)
        atomicExch(a.scan_status + tile, lb_word(epoch, tile == 0 ? LB_INC : LB_AGG, tot));
      const unsigned long long prefix = look_back(a, epoch, tile);
      if (threadIdx.x == 0) {
        const unsigned long long T = lb_sum(prefix, tot);  // elements up to this tile
        if (tile > 0) atomicExch(a.scan_status + tile, lb_word(epoch, LB_INC, T));
        s_prefix = prefix;
        if (tile + 1 == ntiles) {
          a.woff[R] = T;
          a.ctr[lvl_slot(int(i), L_T)] = T;
          if (T <= a.seg_cap)
            a.tile_row[(T + EXPAND_TILE - 1) / EXPAND_TILE] = uint32_t(R - 1);
          else if (a.lane)
            atomicOr(&a.ctr[C_ERR], (unsigned long long)ERR_OVERFLOW);
          if (!a.lane && T > a.t_limit) a.ctr[C_STOP] = i + 1;
        }
      }
    }
    unsigned long long o = ex;
    for (int j = 0; j < 4; ++j) {
      s_off[threadIdx.x * 4 + j] = o;
      o += v[j];
    }
    __syncthreads();
    const unsigned long long prefix = s_prefix;
    for (uint32_t x = threadIdx.x; x < WS_ROWS; x += 256) {
      const uint64_t r = uint64_t(tile) * WS_ROWS + x;
      if (r < R) a.woff[r] = prefix + s_off[x];
    }
    // expand tiles that begin among these rows' elements: the last row that
    // starts at or before their first element
    const uint64_t j1 = (prefix + tot + EXPAND_TILE - 1) / EXPAND_TILE;
    for (uint64_t j = (prefix + EXPAND_TILE - 1) / EXPAND_TILE + threadIdx.x; j < j1; j += 256) {
      if (j * EXPAND_TILE >= a.seg_cap) break;
      const unsigned long long t = j * EXPAND_TILE - prefix;
      uint32_t lo = 0;
      for (uint32_t d = WS_ROWS / 2; d > 0; d >>= 1)
        if (s_off[lo + d] <= t) lo += d;
      a.tile_row[j] = uint32_t(min(uint64_t(tile) * WS_ROWS + lo, R - 1));
    }
    if (ntiles <= gridDim.x) break;  // no block takes a second tile
    __syncthreads();                 // s_off and s_prefix are written again
  }
  bal = warp_sum(bal);
  balc = warp_sum(balc);
  if ((threadIdx.x & 31) == 0 && (bal | balc)) {
    atomicAdd(&a.ctr[C_BALG], bal);
    atomicAdd(&a.ctr[C_BALGC], balc);
  }
}

// End of one query on a lane: its count, survivors per prefix length and
// error bits go to the batch arrays (entry q), and the lane's per-query state
// is cleared for the next query.  A query past its element budget reports
// UINT64_MAX.
__global__ void k_lane_done(unsigned long long* ctr, unsigned long long* counts,
                            unsigned long long* lvl, unsigned long long* qel,
                            unsigned long long budget, uint32_t q,
                            unsigned long long next_elems, unsigned long long* out_counts, unsigned long long* out_lvl,
                            unsigned long long* out_err, unsigned long long* out_balg) {
  const uint32_t t = threadIdx.x;
  if (t <= MAXK) {
    out_lvl[uint64_t(q) * (MAXK + 1) + t] = lvl[t];
    lvl[t] = 0;
  }
  __syncwarp();
  if (t == 0) {
    out_counts[q] = (budget && qel[0] > budget) ? ~0ull : counts[0];
    out_err[q] = ctr[C_ERR];
    out_balg[2ull * q] = ctr[C_BALG];
    out_balg[2ull * q + 1] = ctr[C_BALGC];
    counts[0] = 0;
    qel[0] = next_elems;  // the next query's level-0 candidates
    ctr[C_ERR] = 0;
    ctr[C_BALG] = 0;
    ctr[C_BALGC] = 0;
  }
  for (int c = C_LVL + int(t); c < C_NUM; c += 32) ctr[c] = 0;
}

__global__ void k_set_u64(unsigned long long* p, unsigned long long v) { *p = v; }

// ---------------------------------------------------------------------------
// Plans
// ---------------------------------------------------------------------------
int build_plan(const DevGraph* dg, const QueryGraph& Q, const uint32_t* order, PlanDev* P) {
  std::memset(P, 0, sizeof(*P));
  const uint32_t k = Q.k;
  P->k = k;
  const bool sym = dg->g.symmetric != 0;
  int clab[MAXK];
  for (uint32_t u = 0; u < k; ++u) clab[u] = dg->stats.compact_label(Q.label_raw[u]);
  for (uint32_t i = 0; i < k; ++i) {
    const uint32_t u = order[i];
    P->perm[i] = u;
    if (clab[u] < 0) P->zero = 1;
    P->label[i] = clab[u] < 0 ? 0 : uint32_t(clab[u]);
  }
  for (uint32_t i = 0; i < k; ++i) {
    const uint32_t u = order[i];
    uint32_t nc = 0;
    for (uint32_t j = 0; j < i; ++j) {
      const uint32_t w = order[j];
      const bool w_to_u = (Q.out_mask[w] >> u) & 1u;  // u in N_out(w)
      const bool u_to_w = (Q.out_mask[u] >> w) & 1u;  // u in N_in(w)
      if (sym) {
        if (w_to_u || u_to_w) P->cons[i][nc++] = j;
      } else {
        if (w_to_u) P->cons[i][nc++] = j;
        if (u_to_w) P->cons[i][nc++] = j | (1u << 8);
      }
      if (Q.label_raw[w] == Q.label_raw[u]) P->samelab[i] |= 1u << j;
    }
    P->ncons[i] = nc;
    if ((Q.out_mask[u] >> u) & 1u) P->selfloop_mask |= 1u << i;
    uint32_t nb0 = sym ? (Q.out_mask[u] | Q.in_mask[u]) : Q.out_mask[u];
    uint32_t nb1 = Q.in_mask[u];
    P->req[0][i] = __builtin_popcount(nb0);
    P->req[1][i] = sym ? 0 : __builtin_popcount(nb1);
    for (uint32_t w = 0; w < k; ++w) {
      if (clab[w] < 0) continue;
      if ((nb0 >> w) & 1u) P->nlbq[0][i][clab[w] >> 5] |= 1u << (clab[w] & 31);
      if (!sym && ((nb1 >> w) & 1u)) P->nlbq[1][i][clab[w] >> 5] |= 1u << (clab[w] & 31);
    }
  }
  const uint32_t kl = k - 1;
  P->last_o1 = (k >= 2 && P->ncons[kl] == 1 && !((P->selfloop_mask >> kl) & 1u)) ? 1u : 0u;
  if (P->last_o1 && k >= 3 && !P->zero) {
    const uint32_t ia = k - 2;
    const uint32_t cb = P->cons[kl][0], ca = P->cons[ia][0];
    if ((cb & 0xFF) == ia && P->ncons[ia] == 1 && !((P->selfloop_mask >> ia) & 1u)) {
      const uint32_t p = ca & 0xFF, da = ca >> 8, db = cb >> 8;
      uint32_t Ia = 0, J = 0;
      for (uint32_t j = 0; j < ia; ++j) {
        if (P->label[j] == P->label[ia]) Ia |= 1u << j;
        if (P->label[j] == P->label[kl]) J |= 1u << j;
      }
      // every j in J must be p with x in N^{rev db}(m_p) <=> x in N^{da}(m_p)
      const bool ok = J == 0 || (J == (1u << p) && (sym || da != db));
      if (ok) {
        P->tail2 = 1;
        P->tail_p = p;
        P->tail_da = da;
        P->tail_db = db;
        P->tail_Ia = Ia;
        P->tail_J = J;
      }
    }
  }
  if (!P->tail2 && P->last_o1 && k >= 3 && !P->zero) {
    // Two final leaves of one anchor: k-2 and k-1 have the same single
    // backward constraint (position and direction), so they are not adjacent.
    const uint32_t ia = k - 2, cb = P->cons[kl][0];
    if (P->ncons[ia] == 1 && P->cons[ia][0] == cb && (cb & 0xFF) < ia &&
        !((P->selfloop_mask >> ia) & 1u)) {
      P->star2 = 1;
      P->star_p = cb & 0xFF;
      P->star_d = cb >> 8;
    }
  }
  if (P->last_o1) {
    const uint32_t cs = P->cons[kl][0];
    const uint32_t ws = order[cs & 0xFF], dir = cs >> 8;
    for (uint32_t m = P->samelab[kl]; m; m &= m - 1) {
      const uint32_t j = __builtin_ctz(m);
      const uint32_t wj = order[j];
      bool g;
      if (sym) g = ((Q.out_mask[ws] >> wj) & 1u) || ((Q.out_mask[wj] >> ws) & 1u);
      else if (dir == 0) g = (Q.out_mask[ws] >> wj) & 1u;  // m(j) in N_out(m(ws))
      else g = (Q.out_mask[wj] >> ws) & 1u;                // m(j) in N_in(m(ws))
      if (g) P->guar[kl] |= 1u << j;
    }
  }
  return MG_OK;
}

static int choose_order(DevGraph* dg, const QueryGraph& Q, const mg_opts& o, uint32_t* order) {
  switch (o.order) {
    case MG_ORDER_REFERENCE:
      order_reference(Q, order);
      return MG_OK;
    case MG_ORDER_STRONG:
      order_strong(Q, dg->stats, order);
      return MG_OK;
    case MG_ORDER_LEARNED: {
      if (!o.model) {
        order_reference(Q, order);
        return MG_OK;
      }
      int rc = ensure_full_stats(dg);
      if (rc) return rc;
      return order_learned(o.model, Q, dg->stats, order);
    }
    case MG_ORDER_GIVEN:
      if (!o.given_order) return set_error(MG_E_ARG, "MG_ORDER_GIVEN without given_order");
      std::memcpy(order, o.given_order, Q.k * 4);
      if (!order_is_permutation(order, Q.k))
        return set_error(MG_E_ARG, "given_order is not a permutation of 0..%u", Q.k - 1);
      return MG_OK;
    default:
      return set_error(MG_E_ARG, "unknown order %d", o.order);
  }
}

// ---------------------------------------------------------------------------
// Host driver: depth-first walk over level chunks
// ---------------------------------------------------------------------------
struct RunResult {
  uint64_t balg = 0, balgc = 0, launches = 0, chunks = 0, elements = 0, expand_launches = 0;
  uint64_t reruns = 0;  // batch queries counted again on the chunked path
  double expand_ms = 0;
  uint64_t surv[MAXK + 2] = {};
  uint64_t emitted = 0;
  bool emit_full = false;  // the emit buffer was too small
  double ms = 0;
};

static inline unsigned grid_for(uint64_t items, unsigned block, unsigned cap) {
  uint64_t g = (items + block - 1) / block;
  return unsigned(std::max<uint64_t>(1, std::min<uint64_t>(g, cap)));
}

// Shape of the expand kernel for what the rows of level i can need: a write
// when the level writes a table, emit rows in emit mode, in-place closing of a
// last position or of a pendant tail when a plan has one right after this
// position.
static int expand_mode(const StepArgs& a, uint32_t i, const PlanDev* plans, uint32_t nplans,
                       bool count_mode, bool writes) {
  bool fused = false, tail = false, emit = false;
  for (uint32_t pi = 0; pi < nplans; ++pi) {
    const PlanDev& p = plans[pi];
    if (count_mode && p.k == i + 2 && p.last_o1) fused = true;
    if (((a.tail_dense && p.tail2) || (a.star && p.star2)) && p.k == i + 3) tail = true;
    if (!count_mode && p.k == i + 1) emit = true;
  }
  // Closed where they are found: a single query's candidates, when the probes
  // that this takes (further constraints and look-ups) fit a row's two slots.
  // Not a tail whose anchor is joined to the candidate and whose position k-2
  // has its label: every candidate would take the slow path there (5.1 ms
  // against 2.9 ms staged over such queries of a batch on R-MAT scale 22).
  if (nplans == 1 && !writes && !emit && fused != tail && a.g.symmetric &&
      (fused || plans[0].tail2)) {
    const PlanDev& p = plans[0];
    const int others = std::max(0, int(p.ncons[i]) - 1);
    bool sure = false;
    if (tail && p.tail_p != i && (p.tail_Ia >> i & 1u))
      for (uint32_t c = 0; c < p.ncons[i]; ++c) sure |= (p.cons[i][c] & 0xFF) == p.tail_p;
    if (!sure && others + __builtin_popcount(direct_sides(p, i, tail)) <= 2)
      return X_DIRECT | X_ONE | (fused ? X_FUSED : X_TAIL) | (others == 0 ? X_ALONE : 0);
  }
  const bool plain = nplans == 1 && !emit && !fused && !tail &&
                     __builtin_popcount(plans[0].samelab[i]) <= 2 &&
                     !((plans[0].selfloop_mask >> i) & 1u) && !(i == 0 && a.root_keep);
  const uint32_t nc = plans[0].ncons[i];
  return (writes ? X_WRITE : 0) | (emit ? X_EMIT : 0) | (fused ? X_FUSED : 0) |
         (tail ? X_TAIL : 0) | (nplans == 1 ? X_ONE : 0) | (plain && nc == 2 ? X_PAIR : 0) |
         (plain && nc == 3 ? X_TRIO : 0);
}

// Launches a kernel that begins with chain_begin / chain_wait behind the kernel
// ahead of it in the stream; `chained`: it need not wait for that one's end to
// be launched.
template <class... Args>
static cudaError_t launch_chained(void (*kernel)(Args...), unsigned grid, unsigned block,
                                  cudaStream_t st, bool chained, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.stream = st;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = chained ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

static cudaError_t launch_expand(const StepArgs& a, int mode, unsigned grid, cudaStream_t st,
                                 bool chained) {
  switch (mode) {
#define MG_X(m) \
  case m:       \
    return launch_chained(k_expand<m>, grid, EXPAND_BLOCK, st, chained, a);
    // a batch's level, by what some query of it does there
    MG_X(0) MG_X(1) MG_X(4) MG_X(5) MG_X(8) MG_X(9) MG_X(12) MG_X(13)
    // one query's level does one of them (emit runs hold one query)
    MG_X(16) MG_X(17) MG_X(18) MG_X(20) MG_X(24)
    MG_X(52) MG_X(56) MG_X(116) MG_X(120) MG_X(144) MG_X(145) MG_X(272) MG_X(273)
#undef MG_X
  }
  return cudaErrorInvalidDeviceFunction;  // no such shape
}

// Tail keys (da, la, db, lb, lp) of the plans that end in a two-position
// pendant tail, their tables of two-hop aggregates over the bucket of l_p (all
// keys of a call share one array of at most kTailEntries entries; a key past it
// sums in place) and the tail fields of `a`.
constexpr uint64_t kTailEntries = 1ull << 29;  // 8 GiB

static int setup_tails(DevGraph* dg, std::vector<PlanDev>& plans, TailStore& ts, cudaStream_t st,
                       StepArgs* a, uint64_t* launches) {
  std::vector<TailKey> keys;
  uint64_t entries = 0;
  uint32_t widest = 0;
  for (PlanDev& p : plans) {
    if (!p.tail2) continue;
    TailKey tk{p.tail_da, p.label[p.k - 2], p.tail_db, p.label[p.k - 1], p.label[p.tail_p], 0, 0};
    uint32_t kid = 0;
    while (kid < keys.size() && std::memcmp(&keys[kid], &tk, 20) != 0) ++kid;
    if (kid == keys.size()) {
      const uint32_t nb = dg->h_bucket_off[tk.lp + 1] - dg->h_bucket_off[tk.lp];
      tk.b0 = dg->h_bucket_off[tk.lp];
      tk.base = entries + nb <= kTailEntries ? entries : ~0ull;
      if (tk.base != ~0ull) {
        entries += nb;
        widest = std::max(widest, nb);
      }
      keys.push_back(tk);
    }
    p.tail_kid = kid;
  }
  if (keys.empty()) return MG_OK;
  if (ts.cap < entries || ts.keys_cap < keys.size()) {
    const uint64_t want = std::max<uint64_t>(entries, ts.cap);
    const uint32_t nk = std::max<uint32_t>(uint32_t(keys.size()), ts.keys_cap);
    MG_CK(cudaStreamSynchronize(st));
    ts.free();
    if (cudaMalloc((void**)&ts.keys, nk * sizeof(TailKey)) != cudaSuccess) {
      cudaGetLastError();
      ts.keys = nullptr;
      return set_error(MG_E_OOM, "tail keys: cudaMalloc failed");
    }
    ts.keys_cap = nk;
    if (cudaMalloc((void**)&ts.agg, want * sizeof(uint4)) == cudaSuccess) {
      ts.cap = want;
    } else {  // no room for tables: every key sums in place
      cudaGetLastError();
      ts.agg = nullptr;
      for (TailKey& tk : keys) tk.base = ~0ull;
      widest = 0;
    }
  }
  MG_CK(cudaMemcpyAsync(ts.keys, keys.data(), keys.size() * sizeof(TailKey),
                        cudaMemcpyHostToDevice, st));
  for (uint32_t k0 = 0; widest && k0 < keys.size(); k0 += 65535) {
    const uint32_t nk = std::min<uint32_t>(uint32_t(keys.size()) - k0, 65535);
    k_tail_table<<<dim3((widest + TA_V - 1) / TA_V, nk), TA_BLOCK, 0, st>>>(dg->g, ts.keys + k0,
                                                                           ts.agg);
    ++*launches;
  }
  MG_CK(cudaGetLastError());
  a->tail_dense = 1;
  a->tail_agg = ts.agg;
  a->tkeys = ts.keys;
  return MG_OK;
}

// Last level a plan expands in count mode: k-1, or k-2 when the last
// position is closed in place, or k-3 when a pendant tail is closed from
// dense aggregates.
static int last_level(const PlanDev& P, bool dense, bool star) {
  int l = int(P.k) - 1;
  if (P.k >= 2 && P.last_o1) l = int(P.k) - 2;
  if ((dense && P.tail2) || (star && P.star2)) l = int(P.k) - 3;
  return l;
}

// Candidates of level 0 (see row_work): the label bucket of the first position,
// or the part of it that the options name.
static uint64_t root_range(const DevGraph* dg, const PlanDev& P, const StepArgs& a,
                           uint32_t* first) {
  const uint64_t b0 = dg->h_bucket_off[P.label[0]];
  const uint64_t size = dg->h_bucket_off[P.label[0] + 1] - b0;
  *first = uint32_t(b0);
  if (P.zero) return 0;
  if (!a.root_end) return size;
  const uint64_t rb = std::min<uint64_t>(a.root_begin, size), re = std::min(a.root_end, size);
  *first = uint32_t(b0 + rb);
  return re > rb ? (re - rb + a.root_step - 1) / a.root_step : 0;
}

// Algorithmic bytes of a level-0 candidate: its id, degree and label bits.
static uint64_t root_charge(const DevGraph* dg) { return 12ull + 4ull * dg->g.W; }

// Upper bound of the elements of a row of level l.
static uint64_t row_bound(const DevGraph* dg, const PlanDev* plans, uint32_t nq, int l) {
  for (uint32_t q = 0; q < nq; ++q)
    if (uint32_t(l) < plans[q].k && plans[q].ncons[l] == 0) return dg->g.n;
  return dg->g.symmetric ? std::max(dg->info.max_degree, 1u) : dg->g.n;
}

static uint64_t bounded_product(uint64_t a, uint64_t b) {
  return b && a > (1ull << 40) / b ? 1ull << 40 : a * b;
}

// Scratch of a walk over the levels.
struct WalkBufs {
  uint64_t cap = 0;  // rows per level table, at most
  const uint64_t* rows = nullptr;  // rows that each table holds now (nullptr: cap)
  Workspace* grow = nullptr;       // whose tables can grow up to cap
  uint32_t* (*col)[MAXK] = nullptr;
  uint32_t** qid = nullptr;  // nullptr: single queries only
  uint64_t** woff = nullptr;
  uint32_t** dstart = nullptr;
  uint8_t** dci = nullptr;
  uint32_t* tile_row = nullptr;
  uint64_t seg = 0;  // elements that tile_row covers
  unsigned long long* status = nullptr;
  uint64_t status_bytes = 0;
  uint32_t* epoch = nullptr;
  unsigned long long* res = nullptr;    // device result block, zeroed
  unsigned long long* h_res = nullptr;  // host mirror: one query's block, or the counters
  cudaEvent_t done = nullptr, ev2 = nullptr, ev3 = nullptr;
};

// Depth-first walk over the level tables.  From a level whose rows are known,
// all deeper levels are queued at once with their sizes on the device (work/scan
// and expand per level, no host in between): a level with more elements than
// its table or the budget allows stops the chain (C_STOP), and the host goes on
// from there, one chunk of that level at a time, each followed by the chain of
// the levels below.  So a query that fits its tables costs one synchronisation,
// and a larger one costs one per chunk.
//
// With a work kernel, three scan kernels, a tile-row kernel and two host waits
// per level, a labelled 4-cycle on a 10,000-vertex graph took 24 launches and
// 312 us; it takes 7 and 120 us.  R-MAT scale 22, 4-clique: 7.3 -> 6.9 ms; 48
// budgeted runs on scale 20: 65 -> 19 ms (a run past its budget on a batch
// lane is not counted again); 256 single queries 128 -> 105 ms.
static int walk_levels(DevGraph* dg, const PlanDev* plans, uint32_t nq, bool count_mode,
                       const mg_opts& o, StepArgs a, WalkBufs& B, RunResult* res) {
  const bool one = nq == 1;
  const unsigned sms = dg->sms;
  cudaStream_t st = dg->stream;
  const bool dense = a.tail_dense != 0, star = a.star != 0;
  // writes[l]: some query can append rows to the level-(l+1) table.
  bool writes[MAXK] = {};
  int last = -1;
  for (uint32_t q = 0; q < nq; ++q) {
    const PlanDev& p = plans[q];
    if (p.zero) continue;
    const int lp = count_mode ? last_level(p, dense, star) : int(p.k) - 1;
    for (int l = 0; l < lp; ++l) writes[l] = true;
    last = std::max(last, lp);
  }
  int mode[MAXK] = {};
  uint64_t widest[MAXK] = {};  // elements of a row, at most
  for (int l = 0; l <= last; ++l) {
    mode[l] = expand_mode(a, uint32_t(l), plans, nq, count_mode, writes[l]);
    widest[l] = row_bound(dg, plans, nq, l);
  }
  a.ctr = B.res;
  a.counts = B.res + C_NUM;
  a.lvl_rows = a.counts + nq;
  a.q_elems = a.lvl_rows + uint64_t(nq) * (MAXK + 1);
  a.seg_cap = B.seg;
  a.tile_row = B.tile_row;
  a.scan_status = B.status;
  a.spin_limit = kSpinLimit;
  a.R = nq;
  unsigned long long* h = B.h_res;
  uint64_t T[MAXK] = {}, cur[MAXK] = {}, elements = 0;
  uint32_t R[MAXK] = {};
  R[0] = nq;
  int rc;

  auto held = [&](int l) { return B.rows ? std::min(B.rows[l], B.cap) : B.cap; };
  auto set_level = [&](int l) {
    a.level = uint32_t(l);
    a.cap_rows = l == 0 ? nq : held(l);
    auto tab = [&](int x) {
      TabPtrs t{};
      for (int j = 0; j < x; ++j) t.col[j] = B.col[x][j];
      t.qid = one ? nullptr : B.qid[x];
      return t;
    };
    a.in = tab(l);
    a.woff = B.woff[l];
    a.dstart = B.dstart[l];
    a.dci = B.dci[l];
    a.out = writes[l] ? tab(l + 1) : TabPtrs{};
    a.out_cap = writes[l] ? held(l + 1) : 0;
    a.out_slot = lvl_slot(l, L_OUT);
    a.tile_slot = lvl_slot(l, L_TILE);
  };
  auto expand = [&](int l, uint64_t bound) -> int {
    if (o.kernel_events && B.ev2) MG_CK(cudaEventRecord(B.ev2, st));
    MG_CK(launch_expand(a, mode[l], grid_for(bound, 256, sms * 4), st, one && a.dev));
    if (o.kernel_events && B.ev2) {
      MG_CK(cudaEventRecord(B.ev3, st));
      MG_CK(cudaEventSynchronize(B.ev3));
      float kms = 0;
      MG_CK(cudaEventElapsedTime(&kms, B.ev2, B.ev3));
      res->expand_ms += kms;
    }
    res->expand_launches++;
    res->launches++;
    return MG_OK;
  };
  auto refuse = [&]() {
    cudaStreamSynchronize(st);
    return set_error(MG_E_LIMIT, "work budget of %llu candidate elements exceeded",
                     (unsigned long long)o.max_elements);
  };
  // Queues levels l0..last, whose first table has at most `rows` rows.
  auto descend = [&](int l0, uint64_t rows) -> int {
    a.dev = 1;
    for (int l = l0; l <= last; ++l) {
      set_level(l);
      a.t_limit = writes[l] ? std::min(held(l + 1), B.seg) : B.seg;
      if (one && o.max_elements) a.t_limit = std::min(a.t_limit, o.max_elements - elements);
      const bool clear = ++*B.epoch > LB_EPOCHS;
      if (clear) {
        MG_CK(cudaMemsetAsync(B.status, 0, B.status_bytes, st));
        *B.epoch = 1;
      }
      MG_CK(launch_chained(k_work_scan, grid_for(rows, WS_ROWS, sms * 4), 256u, st,
                           one && l > l0 && !clear, a, *B.epoch));
      res->launches++;
      const uint64_t bound = std::min(bounded_product(rows, widest[l]), a.t_limit);
      if (int r = expand(l, bound)) return r;
      rows = bound;
    }
    return MG_OK;
  };
  // Waits for what is queued and takes over the sizes of levels l0..last, which
  // ran to their end, or up to the one that stopped (returned in *stop).
  auto settle = [&](int l0, int* stop) -> int {
    if (B.done) MG_CK(cudaEventRecord(B.done, st));
    MG_CK(cudaMemcpyAsync(h, B.res, (one ? res_words(1) : C_NUM) * 8, cudaMemcpyDeviceToHost, st));
    MG_CK(cudaStreamSynchronize(st));
    MG_CK(cudaGetLastError());
    if (h[C_ERR] & ERR_TIMEOUT) return set_error(MG_E_TIMEOUT, "a device wait gave up");
    if (a.emit_cap && h[C_EMIT] > a.emit_cap) {
      res->emit_full = true;
      return set_error(MG_E_CUDA, "more matches than the emit buffer holds");
    }
    if (h[C_ERR] & ERR_OVERFLOW) return set_error(MG_E_CUDA, "device table overflow");
    *stop = -1;
    const uint64_t budget = one && o.max_elements ? o.max_elements : ~0ull;
    for (int l = l0; l <= last; ++l) {
      R[l] = l == 0 ? nq : uint32_t(h[lvl_slot(l - 1, L_OUT)]);
      T[l] = h[lvl_slot(l, L_T)];
      if (h[C_STOP] == uint64_t(l) + 1) {
        cur[l] = 0;
        *stop = l;
        if (T[l] > budget - elements) return refuse();
        if (T[l] >= LB_MAX)
          return set_error(MG_E_LIMIT, "a level of 2^%d or more candidate elements",
                           LB_VALUE_BITS);
        return MG_OK;
      }
      if (T[l] > budget - elements) return refuse();
      cur[l] = T[l];
      elements += T[l];
      res->chunks += T[l] > 0;
    }
    return MG_OK;
  };

  int top = -1;
  bool waited = false;
  if (B.grow) {
    if (!one && (rc = ensure_level(B.grow, 0, nq))) return rc;
    for (int l = 1; l <= last; ++l)
      if ((rc = ensure_level(B.grow, l, std::min(B.cap, kFirstRows)))) return rc;
  }
  if (!one) k_iota<<<grid_for(nq, 256, 1024), 256, 0, st>>>(B.qid[0], nq);
  if (one && last >= 0) {
    T[0] = a.T0 = root_range(dg, plans[0], a, &a.root_first);
    res->balg += T[0] * root_charge(dg);
    res->balgc += T[0] * root_charge(dg);
    top = T[0] ? 0 : -1;
  } else if (last >= 0) {
    if ((rc = descend(0, nq))) return rc;
    if ((rc = settle(0, &top))) return rc;
    waited = true;
  }
  while (top >= 0) {
    if (cur[top] >= T[top]) {
      --top;
      continue;
    }
    const uint64_t t0 = cur[top];
    if (writes[top] && B.grow && held(top + 1) < std::min(T[top] - t0, B.cap)) {
      // The next table grows to what this level needs (nothing below this level
      // is in use, the stream is idle); without memory the level is chunked.
      uint64_t want = kFirstRows;
      while (want < T[top] - t0 && want < B.cap) want <<= 1;
      want = std::min(want, B.cap);
      if (ensure_level(B.grow, top + 1, want) &&
          (rc = ensure_level(B.grow, top + 1, std::min(B.cap, kFirstRows))))
        return rc;
      clear_error();
    }
    const uint64_t t1 = writes[top] ? std::min(T[top], t0 + held(top + 1)) : T[top];
    if (one && o.max_elements && t1 - t0 > o.max_elements - elements) return refuse();
    elements += t1 - t0;
    if (waited)  // the slots of this level and below
      MG_CK(cudaMemsetAsync(B.res + lvl_slot(top, 0), 0, (C_NUM - lvl_slot(top, 0)) * 8, st));
    set_level(top);
    a.dev = 0;
    for (uint64_t s0 = t0; s0 < t1; s0 += B.seg) {
      a.t0 = s0;
      a.t1 = std::min(t1, s0 + B.seg);
      if (!(one && top == 0)) {
        const uint32_t ntiles = uint32_t((a.t1 - s0 + EXPAND_TILE - 1) / EXPAND_TILE);
        k_tile_rows<<<grid_for(uint64_t(ntiles) + 1, 256, sms * 16), 256, 0, st>>>(
            B.woff[top], R[top], s0, a.t1, ntiles, B.tile_row);
        res->launches++;
      }
      if (s0 > t0) MG_CK(cudaMemsetAsync(B.res + a.tile_slot, 0, 8, st));
      if ((rc = expand(top, a.t1 - s0))) return rc;
    }
    res->chunks++;
    cur[top] = t1;
    if ((rc = descend(top + 1, t1 - t0))) return rc;
    int stop;
    if ((rc = settle(top + 1, &stop))) return rc;
    waited = true;
    if (stop >= 0) top = stop;
  }
  if (!waited) {  // nothing to expand
    int stop;
    last = -1;
    if ((rc = settle(0, &stop))) return rc;
  }
  res->elements = elements;
  res->balg += h[C_BALG];
  res->balgc += h[C_BALGC];
  res->emitted = h[C_EMIT];
  return MG_OK;
}

static int run_levels(DevGraph* dg, std::vector<PlanDev> plans, bool count_mode,
                      const RowBuf* emit, const mg_opts& o, uint64_t* counts_out,
                      RunResult* res, uint64_t* lvl_rows_out = nullptr) {
  const uint32_t nq = uint32_t(plans.size());
  uint32_t kmax = 1;
  for (auto& p : plans) kmax = std::max(kmax, p.k);
  // Default rows per level chunk: scaled with the graph so small graphs do
  // not reserve gigabytes of scratch; chunking keeps larger results exact.
  uint64_t auto_cap = 1ull << 16;
  while (auto_cap < kDefaultCap && auto_cap < 4 * (uint64_t(dg->g.n) + dg->info.m_out))
    auto_cap <<= 1;
  uint64_t cap = o.chunk_rows ? o.chunk_rows : auto_cap;
  cap = std::max<uint64_t>(cap, 1);
  if (cap > (1ull << 31)) return set_error(MG_E_ARG, "chunk_rows above 2^31");
  if (o.mem_budget_bytes) {
    uint64_t per_row = 0;
    for (uint32_t l = 1; l < kmax; ++l) per_row += level_row_bytes(int(l));
    if (per_row && cap * per_row > o.mem_budget_bytes) {
      cap = o.mem_budget_bytes / per_row;
      if (cap == 0) return set_error(MG_E_OOM, "memory budget below one row per level");
    }
  }
  int rc = ensure_ws(dg, cap, nq);
  if (rc) return rc;
  Workspace* ws = dg->ws;
  if (o.mem_budget_bytes) {  // tables of earlier calls count too
    const uint32_t mask = tables_to_free(ws->rows, MAXK, int(kmax), cap, o.mem_budget_bytes,
                                         [](int l) { return level_row_bytes(l); });
    for (int l = 0; l < MAXK; ++l)
      if (mask >> l & 1u) {
        cudaFree(ws->block[l]);
        ws->block[l] = nullptr;
        ws->rows[l] = 0;
      }
  }
  cudaStream_t st = dg->stream;
  const bool batch = nq > 1;
  MG_CK(cudaEventRecord(ws->ev0, st));
  MG_CK(cudaMemsetAsync(ws->res, 0, res_words(nq) * 8, st));

  StepArgs a;
  std::memset(&a, 0, sizeof(a));
  a.g = dg->g;
  a.plans = ws->plans;
  a.q_budget = batch ? o.max_elements : 0;  // batch: per-query budget
  a.count_mode = count_mode ? 1u : 0u;
  a.filters = o.filters & MG_FILTER_ALL;
  a.grab = o.grab;
  a.nq = nq;
  if (emit) {
    for (int j = 0; j < MAXK; ++j) a.emit_col[j] = emit->col[j];
    a.emit_key = emit->packed ? emit->key_a : nullptr;
    a.emit_k = emit->k;
    a.emit_bits = emit->bits;
    a.emit_cap = emit->cap;
  }
  a.root_step = o.root_step > 1 ? o.root_step : 1u;
  a.probe_min = o.probe_min ? o.probe_min : kProbeMin;
  if (o.root_end || a.root_step > 1) {
    a.root_begin = o.root_begin;
    a.root_end = o.root_end ? o.root_end : ~0ull;
  }
  if (o.matrix_filter && !batch && !plans[0].zero) {
    const uint64_t words = (uint64_t(dg->g.n) + 31) / 32;
    if (ws->root_keep_words < words) {
      ws->root_keep_words = 0;
      if ((rc = ws_alloc((void**)&ws->root_keep, words * 4))) return rc;
      ws->root_keep_words = words;
    }
    if ((rc = matrix_filter_roots(o.matrix_filter, dg, plans[0].perm[0], plans[0].label[0],
                                  ws->root_keep, st)))
      return rc;
    a.root_keep = ws->root_keep;
    res->launches++;
  }
  // Pendant tails counted in closed form (count mode): the tables of two-hop
  // aggregates of their keys, shared by every query of the call.
  if (count_mode && o.no_tail != 1) {
    if ((rc = setup_tails(dg, plans, ws->tails, st, &a, &res->launches))) return rc;
  }
  a.star = count_mode && o.no_tail != 1;
  if (batch) {
    MG_CK(cudaMemcpyAsync(ws->plans, plans.data(), nq * sizeof(PlanDev), cudaMemcpyHostToDevice,
                          st));
  } else {
    *ws->h_plan = plans[0];
    MG_CK(cudaMemcpyAsync(ws->plans, ws->h_plan, sizeof(PlanDev), cudaMemcpyHostToDevice, st));
  }

  WalkBufs B;
  B.cap = cap;
  B.rows = ws->rows;
  B.grow = ws;
  B.col = ws->col;
  B.qid = ws->qid;
  B.woff = ws->woff;
  B.dstart = ws->dstart;
  B.dci = ws->dci;
  B.tile_row = ws->tile_row;
  B.seg = kSegment;
  B.status = ws->status;
  B.status_bytes = ws->status_bytes;
  B.epoch = &ws->epoch;
  B.res = ws->res;
  B.h_res = ws->h_res;
  B.done = ws->ev1;
  B.ev2 = ws->ev2;
  B.ev3 = ws->ev3;
  rc = walk_levels(dg, plans.data(), nq, count_mode, o, a, B, res);
  float ms = 0;
  if (rc == MG_OK || res->emit_full) MG_CK(cudaEventElapsedTime(&ms, ws->ev0, ws->ev1));
  res->ms = ms;
  if (rc) {
    cudaStreamSynchronize(st);
    return rc;
  }
  const unsigned long long *cnt = ws->h_res + C_NUM, *lvl = cnt + nq, *qel = lvl + MAXK + 1;
  std::vector<unsigned long long> all;
  if (batch) {
    all.resize(res_words(nq) - C_NUM);
    MG_CK(cudaMemcpyAsync(all.data(), ws->res + C_NUM, all.size() * 8, cudaMemcpyDeviceToHost, st));
    MG_CK(cudaStreamSynchronize(st));
    cnt = all.data();
    lvl = cnt + nq;
    qel = lvl + uint64_t(nq) * (MAXK + 1);
  }
  for (uint32_t q = 0; q < nq; ++q)  // over budget: unknown
    counts_out[q] = a.q_budget && qel[q] > a.q_budget ? ~0ull : cnt[q];
  if (lvl_rows_out)
    for (uint64_t x = 0; x < uint64_t(nq) * (MAXK + 1); ++x) lvl_rows_out[x] = lvl[x];
  for (int x = 0; x <= MAXK; ++x) res->surv[x] = lvl[x];
  return MG_OK;
}

// ---------------------------------------------------------------------------
// Entry-point bodies
// ---------------------------------------------------------------------------
static mg_opts resolve_opts(const mg_opts* o) {
  mg_opts r;
  mg_opts_default(&r);
  if (o) r = *o;
  return r;
}

// Checks that do not depend on the query or the graph.
static int check_opts(const mg_opts& o) {
  if (o.root_end && o.root_begin > o.root_end)
    return set_error(MG_E_ARG, "root_begin > root_end");
  return MG_OK;
}

static void fill_stats(mg_stats* st, const PlanDev& P, const RunResult& res, uint64_t count) {
  if (!st) return;
  std::memset(st, 0, sizeof(*st));
  st->k = P.k;
  for (uint32_t i = 0; i < P.k; ++i) st->order[i] = P.perm[i];
  for (uint32_t i = 1; i <= P.k && i <= MAXK; ++i) st->level_rows[i] = res.surv[i];
  st->level_rows[P.k] = count;
  st->balg_bytes = res.balg;
  st->balg_count_bytes = res.balgc;
  st->device_ms = res.ms;
  st->launches = res.launches;
  st->chunks = res.chunks;
  st->elements = res.elements;
  st->expand_ms = res.expand_ms;
  st->expand_launches = res.expand_launches;
}

// Where emitted rows go: a caller's buffer of cap_rows rows, or memory that the
// caller hands out once the number of rows is known.
struct RowSink {
  uint64_t cap_rows = 0;
  uint32_t* buffer = nullptr;
  mg_rows_alloc alloc = nullptr;
  void* ctx = nullptr;
  uint32_t* rows(uint64_t n) const { return alloc ? alloc(ctx, n) : buffer; }
};

static int prepare(DevGraph* dg, const mg_csr_view* q, const mg_opts& o, PlanDev* P) {
  int rc = check_opts(o);
  if (rc) return rc;
  QueryGraph Q;
  rc = normalise_query(q, &Q);
  if (rc) return rc;
  uint32_t order[MAXK];
  if ((rc = choose_order(dg, Q, o, order))) return rc;
  return build_plan(dg, Q, order, P);
}

int subiso_count(DevGraph* dg, const mg_csr_view* q, const mg_opts* opts, uint64_t* count,
                 mg_stats* st) {
  const mg_opts o = resolve_opts(opts);
  PlanDev P;
  int rc = prepare(dg, q, o, &P);
  if (rc) return rc;
  std::vector<PlanDev> plans(1, P);
  RunResult res;
  uint64_t c = 0;
  if ((rc = run_levels(dg, plans, true, nullptr, o, &c, &res))) return rc;
  *count = c;
  fill_stats(st, P, res, c);
  return MG_OK;
}

// Lays out an emit buffer for `cap` rows in the graph's emit block, which grows
// as needed and is given back by trim_emit when it is large: 256 MiB hold 2^22
// rows of up to 4 ids whatever their bits.
constexpr uint64_t kEmitKeep = 1ull << 28;

static uint32_t id_bits(const DevGraph* dg) {
  uint32_t bits = 1;
  while (bits < 32 && dg->max_gid >> bits) ++bits;
  return bits;
}

static int emit_buffer(DevGraph* dg, uint32_t k, uint64_t cap, RowBuf* B) {
  const uint32_t bits = id_bits(dg);
  const uint64_t bytes = B->carve(nullptr, k, bits, cap);
  if (dg->emit_bytes < bytes) {
    MG_CK(cudaStreamSynchronize(dg->stream));
    cudaFree(dg->emit_mem);
    dg->emit_mem = nullptr;
    dg->emit_bytes = 0;
    if (cudaMalloc((void**)&dg->emit_mem, bytes) != cudaSuccess) {
      cudaGetLastError();
      dg->emit_mem = nullptr;
      return set_error(MG_E_OOM, "emit buffer: cudaMalloc(%llu) failed",
                       (unsigned long long)bytes);
    }
    dg->emit_bytes = bytes;
  }
  B->carve(dg->emit_mem, k, bits, cap);
  return MG_OK;
}

static void trim_emit(DevGraph* dg) {
  if (dg->emit_bytes <= kEmitKeep) return;
  cudaFree(dg->emit_mem);
  dg->emit_mem = nullptr;
  dg->emit_bytes = 0;
}

// Matches are emitted at once into a buffer for the caller's rows (emit_room);
// only a query with more of them, or a caller with room for very many, is
// counted first and emitted into a buffer of that size.  With a count before
// every emit, nine allocations a call and the column-wise sort, an emit of some
// thousand rows on a 10,000-vertex graph took 1,384 us; it takes 185 us.
// Triangles of R-MAT scale 18 (16,000 to 2 million rows): 2.1 -> 0.9 ms.
int subiso_emit(DevGraph* dg, const mg_csr_view* q, const mg_opts* opts, const RowSink& sink,
                uint64_t* n_rows, mg_stats* st) {
  const mg_opts o = resolve_opts(opts);
  PlanDev P;
  int rc = prepare(dg, q, o, &P);
  if (rc) return rc;
  std::vector<PlanDev> plans(1, P);
  cudaStream_t s = dg->stream;
  RunResult tried, counted, res;  // an attempt, a count, the pass that gave the rows
  RowBuf eb;
  uint64_t c = 0, unused = 0;
  const uint64_t limit = o.mem_budget_bytes ? std::min(o.mem_budget_bytes, kEmitKeep) : kEmitKeep;
  const uint64_t room = emit_room(
      !sink.alloc, sink.cap_rows, uint64_t(dg->g.n) + dg->info.m_out, limit, dg->emit_bytes,
      [&](uint64_t rows) { return RowBuf().carve(nullptr, P.k, id_bits(dg), rows); });
  if (room) rc = emit_buffer(dg, P.k, room, &eb);
  const bool no_room = !room || rc == MG_E_OOM;
  if (!no_room && rc == MG_OK) {
    rc = run_levels(dg, plans, false, &eb, o, &unused, &res);
    if (rc == MG_OK) c = *n_rows = res.emitted;
    else if (res.emit_full) std::swap(tried, res);
  }
  if (no_room || tried.emit_full) {
    // More matches than the buffer holds, or no memory for it: counted first.
    // Every other failure (a refused budget, a wait that gave up) is the call's.
    clear_error();
    rc = run_levels(dg, plans, true, nullptr, o, &c, &counted);
    if (rc == MG_OK) *n_rows = c;
    if (rc == MG_OK && c >= (1ull << 31))
      rc = set_error(MG_E_LIMIT, "%llu matches: emit supports fewer than 2^31 rows",
                     (unsigned long long)c);
    if (rc == MG_OK) rc = emit_buffer(dg, P.k, c, &eb);
    if (rc == MG_OK) rc = run_levels(dg, plans, false, &eb, o, &unused, &res);
    if (rc == MG_OK && res.emitted != c)
      rc = set_error(MG_E_CUDA, "emit pass produced %llu rows, count pass %llu",
                     (unsigned long long)res.emitted, (unsigned long long)c);
    res.balg = counted.balg;
    res.balgc = counted.balgc;
  }
  if (rc == MG_OK) {
    const uint64_t n_copy = std::min(c, sink.cap_rows);
    uint32_t* rows = sink.rows(n_copy);
    if (n_copy && !rows) rc = set_error(MG_E_OOM, "no memory for %llu rows",
                                        (unsigned long long)n_copy);
    else rc = sort_rows(eb, c, n_copy, rows, dg->sms, kSpinLimit, s);
  }
  cudaStreamSynchronize(s);
  trim_emit(dg);
  if (rc) return rc;
  res.ms += tried.ms + counted.ms;
  res.launches += tried.launches + counted.launches;
  fill_stats(st, P, res, c);
  if (c > sink.cap_rows)
    return set_error(MG_E_CAPACITY, "%llu matches, %llu rows written",
                     (unsigned long long)c, (unsigned long long)sink.cap_rows);
  return MG_OK;
}

// ---------------------------------------------------------------------------
// Batch lane pipeline
//
// Each query of a batch runs as a fixed sequence of launches (level 0: the
// expand; every level after it: the single-pass work/scan and the expand) whose
// kernels read every size from device counters, so nothing returns to the host
// between levels or between queries.  Queries are dealt round-robin to `lanes`
// streams that run concurrently; each lane owns level tables of `cap` rows.
// The host waits once per batch; a query whose rows or elements did not fit
// its lane (ERR_OVERFLOW) is counted again on the chunked path, which has no
// size limit.
// ---------------------------------------------------------------------------
struct Lane {
  cudaStream_t st = nullptr;
  unsigned long long *ctr = nullptr, *counts = nullptr, *lvl = nullptr, *qel = nullptr;
  unsigned long long* status = nullptr;  // look-back words of the work/scan kernel
  uint32_t* tile_row = nullptr;
  uint32_t* col[MAXK][MAXK] = {};
  uint64_t* woff[MAXK] = {};
  uint32_t* dstart[MAXK] = {};
  uint8_t* dci[MAXK] = {};
  uint32_t epoch = 0;
};

struct LaneSet {
  uint64_t cap = 0, seg_cap = 0;
  uint32_t kmax = 0;
  std::vector<Lane> lanes;
  std::vector<void*> allocs;
  unsigned long long *r_counts = nullptr, *r_lvl = nullptr, *r_err = nullptr, *r_balg = nullptr;
  PlanDev* plans = nullptr;
  uint32_t nq_cap = 0;  // queries that plans and the results hold
  TailStore tails;
  cudaEvent_t ev_start = nullptr, ev_end = nullptr;
};

constexpr uint64_t kLaneCap = 1ull << 20;     // rows per lane level table
constexpr uint64_t kLaneSegment = 1ull << 30; // elements per lane expand launch
constexpr uint32_t kLanes = 8;

void free_lanes(LaneSet* ls) {
  if (!ls) return;
  for (Lane& l : ls->lanes)
    if (l.st) cudaStreamDestroy(l.st);
  for (void* p : ls->allocs) cudaFree(p);
  for (void* p : {(void*)ls->plans, (void*)ls->r_counts, (void*)ls->r_lvl, (void*)ls->r_err,
                  (void*)ls->r_balg})
    cudaFree(p);
  ls->tails.free();
  if (ls->ev_start) cudaEventDestroy(ls->ev_start);
  if (ls->ev_end) cudaEventDestroy(ls->ev_end);
  delete ls;
}

static int lane_alloc(LaneSet* ls, void** p, size_t bytes) {
  *p = nullptr;
  cudaError_t e = cudaMalloc(p, std::max<size_t>(bytes, 16));
  if (e != cudaSuccess) {
    cudaGetLastError();
    *p = nullptr;
    return set_error(MG_E_OOM, "lane scratch: cudaMalloc(%zu) failed: %s", bytes,
                     cudaGetErrorString(e));
  }
  ls->allocs.push_back(*p);
  return MG_OK;
}

static int ensure_lanes(DevGraph* dg, uint32_t nl, uint64_t cap, uint32_t kmax) {
  if (dg->lanes &&
      (dg->lanes->lanes.size() != nl || dg->lanes->cap != cap || dg->lanes->kmax < kmax)) {
    cudaDeviceSynchronize();
    free_lanes(dg->lanes);
    dg->lanes = nullptr;
  }
  if (dg->lanes) return MG_OK;
  // Built aside: the graph never keeps a set of lanes that is not complete.
  std::unique_ptr<LaneSet, void (*)(LaneSet*)> made(new LaneSet(), free_lanes);
  LaneSet* ls = made.get();
  ls->cap = cap;
  ls->seg_cap = kLaneSegment;
  ls->kmax = std::max<uint32_t>(kmax, 8);
  MG_CK(cudaEventCreateWithFlags(&ls->ev_start, cudaEventDisableTiming));
  MG_CK(cudaEventCreateWithFlags(&ls->ev_end, cudaEventDisableTiming));
  ls->lanes.resize(nl);
  int rc;
  for (Lane& L : ls->lanes) {
    MG_CK(cudaStreamCreateWithFlags(&L.st, cudaStreamNonBlocking));
    const uint64_t ntiles = cap / WS_ROWS + 2;
    // All arrays of a lane in one block: measured first, then carved.
    unsigned char* p = nullptr;
    for (int pass = 0; pass < 2; ++pass) {
      uint64_t off = 0;
      auto take = [&](auto** array, uint64_t bytes) {
        if (p) *array = reinterpret_cast<std::remove_reference_t<decltype(**array)>*>(p + off);
        off += (bytes + 255) & ~uint64_t(255);
      };
      take(&L.ctr, C_NUM * 8);
      take(&L.counts, 8);
      take(&L.lvl, (MAXK + 1) * 8);
      take(&L.qel, 8);
      take(&L.status, ntiles * 8);
      take(&L.tile_row, (ls->seg_cap / EXPAND_TILE + 2) * 4);
      for (uint32_t l = 0; l < ls->kmax; ++l) {
        const uint64_t rows = l == 0 ? 1 : cap;
        for (uint32_t j = 0; j < l; ++j) take(&L.col[l][j], rows * 4);
        take(&L.woff[l], (rows + 1) * 8);
        take(&L.dstart[l], rows * 4);
        take(&L.dci[l], rows);
      }
      if (pass == 0 && (rc = lane_alloc(ls, (void**)&p, off))) return rc;
    }
    MG_CK(cudaMemsetAsync(L.status, 0, ntiles * 8, L.st));
  }
  dg->lanes = made.release();
  return MG_OK;
}

// Plans and results of nq queries of a batch.
static int ensure_lane_queries(LaneSet* ls, uint32_t nq) {
  int rc;
  if (ls->nq_cap >= nq) return MG_OK;
  ls->nq_cap = 0;
  if ((rc = ws_alloc((void**)&ls->plans, uint64_t(nq) * sizeof(PlanDev)))) return rc;
  if ((rc = ws_alloc((void**)&ls->r_counts, uint64_t(nq) * 8))) return rc;
  if ((rc = ws_alloc((void**)&ls->r_lvl, uint64_t(nq) * (MAXK + 1) * 8))) return rc;
  if ((rc = ws_alloc((void**)&ls->r_err, uint64_t(nq) * 8))) return rc;
  if ((rc = ws_alloc((void**)&ls->r_balg, uint64_t(nq) * 16))) return rc;
  ls->nq_cap = nq;
  return MG_OK;
}

static int subiso_batch_lanes(DevGraph* dg, std::vector<PlanDev>& plans, const mg_opts& o,
                              uint64_t* counts_out, uint64_t* level_rows_out, RunResult* res) {
  const uint32_t nq = uint32_t(plans.size());
  uint32_t kmax = 1;
  for (auto& p : plans) kmax = std::max(kmax, p.k);
  const uint32_t nl = o.lanes ? o.lanes : kLanes;
  if (nl > 64) return set_error(MG_E_ARG, "lanes=%u: at most 64", nl);
  uint64_t cap = o.chunk_rows ? o.chunk_rows : kLaneCap;
  if (cap > (1ull << 31)) return set_error(MG_E_ARG, "chunk_rows above 2^31");
  int rc = ensure_lanes(dg, nl, cap, kmax);
  if (rc) return rc;
  LaneSet* ls = dg->lanes;
  cudaStream_t st = dg->stream;
  const unsigned sms = dg->sms;

  if ((rc = ensure_lane_queries(ls, nq))) return rc;
  Workspace* ws = dg->ws;  // timing events live with the graph's workspace
  if (!ws && (rc = ensure_ws(dg, 1ull << 16, 1))) return rc;
  ws = dg->ws;
  MG_CK(cudaEventRecord(ws->ev0, st));
  StepArgs a;
  std::memset(&a, 0, sizeof(a));
  // Pendant tails closed from tables of two-hop aggregates (filled on the graph's
  // stream before the lanes start).
  if (o.no_tail != 1) {
    if ((rc = setup_tails(dg, plans, ls->tails, st, &a, &res->launches))) return rc;
  } else {
    for (PlanDev& p : plans) p.tail2 = 0;
  }
  MG_CK(cudaMemcpyAsync(ls->plans, plans.data(), uint64_t(nq) * sizeof(PlanDev),
                        cudaMemcpyHostToDevice, st));
  MG_CK(cudaEventRecord(ls->ev_start, st));

  a.g = dg->g;
  a.count_mode = 1;
  a.star = o.no_tail != 1;
  a.filters = o.filters & MG_FILTER_ALL;
  a.grab = o.grab;
  a.root_step = 1;
  a.probe_min = o.probe_min ? o.probe_min : kProbeMin;
  a.q_budget = o.max_elements;
  a.lane = a.dev = 1;
  a.cap_rows = cap;
  a.seg_cap = ls->seg_cap;
  a.t_limit = ls->seg_cap;
  a.spin_limit = kSpinLimit;
  a.nq = a.R = 1;
  // Level-0 candidates of every query: the elements its budget is charged
  // with before the lane starts.
  std::vector<uint64_t> t0(nq);
  std::vector<uint32_t> first(nq);
  for (uint32_t j = 0; j < nq; ++j) t0[j] = root_range(dg, plans[j], a, &first[j]);
  for (uint32_t l = 0; l < nl; ++l) {
    Lane& L = ls->lanes[l];
    MG_CK(cudaStreamWaitEvent(L.st, ls->ev_start, 0));
    MG_CK(cudaMemsetAsync(L.ctr, 0, C_NUM * 8, L.st));
    MG_CK(cudaMemsetAsync(L.counts, 0, 8, L.st));
    MG_CK(cudaMemsetAsync(L.lvl, 0, (MAXK + 1) * 8, L.st));
    k_set_u64<<<1, 1, 0, L.st>>>(L.qel, l < nq ? t0[l] : 0ull);
  }
  for (uint32_t j = 0; j < nq; ++j) {
    Lane& L = ls->lanes[j % nl];
    const PlanDev& P = plans[j];
    a.plans = ls->plans + j;
    a.ctr = L.ctr;
    a.counts = L.counts;
    a.lvl_rows = L.lvl;
    a.q_elems = L.qel;
    a.scan_status = L.status;
    a.tile_row = L.tile_row;
    int last = P.zero ? -1 : last_level(P, a.tail_dense != 0, a.star != 0);
    if (lane_start(t0[j], o.max_elements, ls->seg_cap) != LaneStart::kRun) last = -1;
    a.T0 = t0[j];
    a.root_first = first[j];
    uint64_t rows = 1;
    for (int l = 0; l <= last; ++l) {
      a.level = uint32_t(l);
      TabPtrs t{};
      for (int c = 0; c < l; ++c) t.col[c] = L.col[l][c];
      a.in = t;
      a.woff = L.woff[l];
      a.dstart = L.dstart[l];
      a.dci = L.dci[l];
      if (l > 0) {
        if (++L.epoch > LB_EPOCHS) {
          MG_CK(cudaMemsetAsync(L.status, 0, (cap / WS_ROWS + 2) * 8, L.st));
          L.epoch = 1;
        }
        k_work_scan<<<grid_for(rows, WS_ROWS, sms * 2), 256, 0, L.st>>>(a, L.epoch);
        res->launches++;
      }
      const bool writes = l < last;
      TabPtrs out{};
      if (writes)
        for (int c = 0; c <= l; ++c) out.col[c] = L.col[l + 1][c];
      a.out = out;
      a.out_cap = writes ? cap : 0;
      a.out_slot = lvl_slot(l, L_OUT);
      a.tile_slot = lvl_slot(l, L_TILE);
      const uint64_t bound =
          l == 0 ? t0[j] : bounded_product(rows, row_bound(dg, &P, 1, l));
      MG_CK(launch_expand(a, expand_mode(a, uint32_t(l), &P, 1, true, writes),
                          grid_for(bound, 256, sms * 4), L.st, false));
      rows = std::min(bound, cap);
      res->launches++;
      res->expand_launches++;
    }
    k_lane_done<<<1, 32, 0, L.st>>>(L.ctr, L.counts, L.lvl, L.qel, o.max_elements, j,
                                   j + nl < nq ? t0[j + nl] : 0ull, ls->r_counts, ls->r_lvl,
                                   ls->r_err, ls->r_balg);
    res->launches++;
  }
  MG_CK(cudaGetLastError());
  for (Lane& L : ls->lanes) {
    MG_CK(cudaEventRecord(ls->ev_end, L.st));
    MG_CK(cudaStreamWaitEvent(st, ls->ev_end, 0));
  }
  MG_CK(cudaEventRecord(ws->ev1, st));
  std::vector<unsigned long long> err(nq), cnt(nq), lv(uint64_t(nq) * (MAXK + 1)),
      balg(uint64_t(nq) * 2);
  MG_CK(cudaMemcpyAsync(cnt.data(), ls->r_counts, uint64_t(nq) * 8, cudaMemcpyDeviceToHost, st));
  MG_CK(cudaMemcpyAsync(err.data(), ls->r_err, uint64_t(nq) * 8, cudaMemcpyDeviceToHost, st));
  MG_CK(cudaMemcpyAsync(lv.data(), ls->r_lvl, lv.size() * 8, cudaMemcpyDeviceToHost, st));
  MG_CK(cudaMemcpyAsync(balg.data(), ls->r_balg, balg.size() * 8, cudaMemcpyDeviceToHost, st));
  MG_CK(cudaStreamSynchronize(st));
  float ms = 0;
  MG_CK(cudaEventElapsedTime(&ms, ws->ev0, ws->ev1));
  res->ms = ms;
  for (uint32_t j = 0; j < nq; ++j) {
    if (lane_start(t0[j], o.max_elements, ls->seg_cap) == LaneStart::kChunked)
      err[j] |= ERR_OVERFLOW;
    if (err[j]) continue;  // charged by its re-run below
    res->balg += balg[2ull * j] + t0[j] * root_charge(dg);
    res->balgc += balg[2ull * j + 1] + t0[j] * root_charge(dg);
  }
  for (uint32_t j = 0; j < nq; ++j) {
    if (err[j] & ERR_TIMEOUT)
      return set_error(MG_E_TIMEOUT, "query %u: a lane's device wait gave up", j);
    if (err[j] & ERR_OVERFLOW) {
      if (o.max_elements && cnt[j] == ~0ull) {
        // The elements that did run already pass its budget.
        for (uint32_t i = 0; i <= MAXK; ++i) lv[uint64_t(j) * (MAXK + 1) + i] = 0;
        res->reruns++;
        continue;
      }
      // Did not fit its lane: count it again on the chunked path.
      std::vector<PlanDev> one(1, plans[j]);
      RunResult r1;
      uint64_t c1 = 0;
      std::vector<uint64_t> l1(MAXK + 1, 0);
      mg_opts o1 = o;
      o1.chunk_rows = 0;
      rc = run_levels(dg, one, true, nullptr, o1, &c1, &r1, l1.data());
      if (rc == MG_E_LIMIT && o.max_elements) {
        // Past the per-query budget on the chunked path as well: unknown, as a
        // query over budget in its lane reports.
        cnt[j] = ~0ull;
        for (uint32_t i = 0; i <= MAXK; ++i) lv[uint64_t(j) * (MAXK + 1) + i] = 0;
        res->reruns++;
        continue;
      }
      if (rc) return rc;
      cnt[j] = c1;
      for (uint32_t i = 0; i <= MAXK; ++i) lv[uint64_t(j) * (MAXK + 1) + i] = l1[i];
      res->balg += r1.balg;
      res->balgc += r1.balgc;
      res->ms += r1.ms;
      res->launches += r1.launches;
      res->reruns++;
    }
  }
  for (uint32_t j = 0; j < nq; ++j) counts_out[j] = cnt[j];
  if (level_rows_out)
    for (uint64_t x = 0; x < lv.size(); ++x) level_rows_out[x] = lv[x];
  return MG_OK;
}

// Self-test of the bounded device wait: one work/scan launch of a lane at
// level 1 over 2 * WS_ROWS rows of the first query vertex's bucket, with the
// counter that hands out tiles already past tile 0, so the block of tile 1
// waits for a predecessor nobody publishes.  The wait gives up after
// `spin_limit` polls and the launch ends with ERR_TIMEOUT in its error word.
static int selftest_wait(DevGraph* dg, const mg_csr_view* q, uint32_t spin_limit,
                         uint64_t* err_bits) {
  PlanDev P;
  mg_opts o;
  mg_opts_default(&o);
  int rc = prepare(dg, q, o, &P);
  if (rc) return rc;
  if (P.k < 2 || P.ncons[1] == 0)
    return set_error(MG_E_ARG, "self-test query needs a second vertex joined to the first");
  if ((rc = ensure_lanes(dg, 1, kLaneCap, std::max<uint32_t>(P.k, 2)))) return rc;
  LaneSet* ls = dg->lanes;
  Lane& L = ls->lanes[0];
  if ((rc = ensure_lane_queries(ls, 1))) return rc;
  cudaStream_t st = L.st;
  const uint64_t rows = 2 * WS_ROWS;
  std::vector<unsigned long long> ctr(C_NUM, 0);
  ctr[lvl_slot(0, L_OUT)] = rows;  // level-1 table holds `rows` rows
  ctr[lvl_slot(1, L_SCAN)] = 1;    // tile 0 of level 1 is never handed out
  MG_CK(cudaMemcpyAsync(ls->plans, &P, sizeof(PlanDev), cudaMemcpyHostToDevice, st));
  MG_CK(cudaMemcpyAsync(L.ctr, ctr.data(), C_NUM * 8, cudaMemcpyHostToDevice, st));
  // every row holds the first vertex of the bucket of position 0
  const uint32_t b0 = dg->h_bucket_off[P.label[0]];
  std::vector<uint32_t> col(rows, b0);
  MG_CK(cudaMemcpyAsync(L.col[1][0], col.data(), rows * 4, cudaMemcpyHostToDevice, st));
  StepArgs a;
  std::memset(&a, 0, sizeof(a));
  a.g = dg->g;
  a.plans = ls->plans;
  a.ctr = L.ctr;
  a.counts = L.counts;
  a.lvl_rows = L.lvl;
  a.q_elems = L.qel;
  a.level = 1;
  a.in.col[0] = L.col[1][0];
  a.woff = L.woff[1];
  a.dstart = L.dstart[1];
  a.dci = L.dci[1];
  a.lane = a.dev = 1;
  a.cap_rows = ls->cap;
  a.seg_cap = a.t_limit = ls->seg_cap;
  a.tile_row = L.tile_row;
  a.scan_status = L.status;
  a.spin_limit = spin_limit;
  a.root_step = 1;
  if (++L.epoch > LB_EPOCHS) {
    MG_CK(cudaMemsetAsync(L.status, 0, (ls->cap / WS_ROWS + 2) * 8, st));
    L.epoch = 1;
  }
  k_work_scan<<<2, 256, 0, st>>>(a, L.epoch);
  MG_CK(cudaGetLastError());
  unsigned long long err = 0;
  MG_CK(cudaMemcpyAsync(&err, L.ctr + C_ERR, 8, cudaMemcpyDeviceToHost, st));
  MG_CK(cudaMemsetAsync(L.ctr, 0, C_NUM * 8, st));
  MG_CK(cudaStreamSynchronize(st));
  *err_bits = err;
  return MG_OK;
}

int subiso_batch(DevGraph* dg, const mg_csr_view* const* qs, uint32_t nq, const mg_opts* opts,
                 uint64_t* counts, mg_stats* st, const uint32_t* orders = nullptr,
                 uint64_t* level_rows = nullptr) {
  const mg_opts o = resolve_opts(opts);
  if (o.matrix_filter)
    return set_error(MG_E_ARG, "matrix_filter applies to single-query count and emit only");
  std::vector<PlanDev> plans(nq);
  std::vector<uint32_t> learned;
  if (!orders && o.order == MG_ORDER_LEARNED && o.model) {
    // One inference launch plans the whole batch.
    int rc = ensure_full_stats(dg);
    if (rc) return rc;
    std::vector<QueryGraph> Q(nq);
    std::vector<const QueryGraph*> qp(nq);
    for (uint32_t i = 0; i < nq; ++i) {
      if ((rc = normalise_query(qs[i], &Q[i])))
        return set_error(rc, "query %u: %s", i, last_error_cstr());
      qp[i] = &Q[i];
    }
    std::vector<std::array<uint32_t, MAXK>> ord;
    if ((rc = order_learned_batch(o.model, qp, dg->stats, ord))) return rc;
    learned.resize(uint64_t(nq) * MAXK);
    for (uint32_t i = 0; i < nq; ++i)
      std::memcpy(&learned[uint64_t(i) * MAXK], ord[i].data(), MAXK * 4);
    orders = learned.data();
  }
  for (uint32_t i = 0; i < nq; ++i) {
    mg_opts oi = o;
    if (orders) {
      oi.order = MG_ORDER_GIVEN;
      oi.given_order = orders + uint64_t(i) * MAXK;
    }
    int rc = prepare(dg, qs[i], oi, &plans[i]);
    if (rc) return set_error(rc, "query %u: %s", i, last_error_cstr());
  }
  RunResult res;
  int rc = o.lanes == MG_LANES_SHARED
               ? run_levels(dg, plans, true, nullptr, o, counts, &res, level_rows)
               : subiso_batch_lanes(dg, plans, o, counts, level_rows, &res);
  if (rc) return rc;
  if (st) {
    std::memset(st, 0, sizeof(*st));
    st->balg_bytes = res.balg;
    st->balg_count_bytes = res.balgc;
    st->device_ms = res.ms;
    st->launches = res.launches;
    st->chunks = res.chunks;
    st->elements = res.elements;
    st->expand_ms = res.expand_ms;
    st->expand_launches = res.expand_launches;
  }
  return MG_OK;
}

}  // namespace mg

// ---------------------------------------------------------------------------
// C-ABI
// ---------------------------------------------------------------------------
extern "C" {

const char* mg_last_error(void) { return mg::last_error_cstr(); }
const char* mg_version(void) { return "mg_subiso 0.1 (sm_100a)"; }

void mg_opts_default(mg_opts* o) {
  if (!o) return;
  std::memset(o, 0, sizeof(*o));
  o->order = MG_ORDER_REFERENCE;
  o->filters = MG_FILTER_ALL;
}

#define MG_ENTRY(dgraph)                                              \
  mg::clear_error();                                                  \
  if (!(dgraph)) return mg::set_error(MG_E_ARG, "null graph handle"); \
  auto* dg = static_cast<mg::DevGraph*>(dgraph);                      \
  std::lock_guard<std::mutex> lock(dg->mu);                           \
  mg::DeviceGuard guard(dg->device)

int mg_plan_order(void* dgraph, const mg_csr_view* q, const mg_opts* opts, uint32_t* order,
                  uint32_t* k) {
  mg::clear_error();
  if (!q || !order || !k) return mg::set_error(MG_E_ARG, "null argument");
  mg::QueryGraph Q;
  int rc = mg::normalise_query(q, &Q);
  if (rc) return rc;
  const mg_opts o = mg::resolve_opts(opts);
  if (!dgraph) {
    if (o.order != MG_ORDER_REFERENCE && o.order != MG_ORDER_GIVEN)
      return mg::set_error(MG_E_ARG, "this order needs a graph handle");
    rc = mg::choose_order(nullptr, Q, o, order);
  } else {
    auto* dg = static_cast<mg::DevGraph*>(dgraph);
    std::lock_guard<std::mutex> lock(dg->mu);
    mg::DeviceGuard guard(dg->device);
    rc = mg::choose_order(dg, Q, o, order);
  }
  if (rc) return rc;
  *k = Q.k;
  return MG_OK;
}

int mg_subiso_count_ex(void* dgraph, const mg_csr_view* q, const mg_opts* opts, uint64_t* count,
                       mg_stats* st) {
  MG_ENTRY(dgraph);
  if (!q || !count) return mg::set_error(MG_E_ARG, "null argument");
  try {
    return mg::subiso_count(dg, q, opts, count, st);
  } catch (const std::bad_alloc&) {
    return mg::set_error(MG_E_OOM, "host allocation failed");
  }
}

int mg_subiso_count(void* dgraph, const mg_csr_view* q, const mg_opts* opts, uint64_t* count) {
  return mg_subiso_count_ex(dgraph, q, opts, count, nullptr);
}

int mg_subiso_emit_ex(void* dgraph, const mg_csr_view* q, const mg_opts* opts, uint32_t* rows,
                      uint64_t cap_rows, uint64_t* n_rows, mg_stats* st) {
  MG_ENTRY(dgraph);
  if (!q || !n_rows || (cap_rows && !rows)) return mg::set_error(MG_E_ARG, "null argument");
  try {
    mg::RowSink sink;
    sink.cap_rows = cap_rows;
    sink.buffer = rows;
    return mg::subiso_emit(dg, q, opts, sink, n_rows, st);
  } catch (const std::bad_alloc&) {
    return mg::set_error(MG_E_OOM, "host allocation failed");
  }
}

int mg_subiso_emit_alloc(void* dgraph, const mg_csr_view* q, const mg_opts* opts,
                         mg_rows_alloc alloc, void* ctx, uint64_t* n_rows, mg_stats* st) {
  MG_ENTRY(dgraph);
  if (!q || !n_rows || !alloc) return mg::set_error(MG_E_ARG, "null argument");
  try {
    mg::RowSink sink;
    sink.cap_rows = ~0ull;
    sink.alloc = alloc;
    sink.ctx = ctx;
    return mg::subiso_emit(dg, q, opts, sink, n_rows, st);
  } catch (const std::bad_alloc&) {
    return mg::set_error(MG_E_OOM, "host allocation failed");
  }
}

int mg_subiso_emit(void* dgraph, const mg_csr_view* q, const mg_opts* opts, uint32_t* rows,
                   uint64_t cap_rows, uint64_t* n_rows) {
  return mg_subiso_emit_ex(dgraph, q, opts, rows, cap_rows, n_rows, nullptr);
}

int mg_subiso_batch_count_ex(void* dgraph, const mg_csr_view* const* qs, uint32_t nq,
                             const mg_opts* opts, uint64_t* counts, mg_stats* st) {
  MG_ENTRY(dgraph);
  if (!qs || !counts || nq == 0) return mg::set_error(MG_E_ARG, "null argument or empty batch");
  try {
    return mg::subiso_batch(dg, qs, nq, opts, counts, st);
  } catch (const std::bad_alloc&) {
    return mg::set_error(MG_E_OOM, "host allocation failed");
  }
}

int mg_subiso_batch_count(void* dgraph, const mg_csr_view* const* qs, uint32_t nq,
                          const mg_opts* opts, uint64_t* counts) {
  return mg_subiso_batch_count_ex(dgraph, qs, nq, opts, counts, nullptr);
}

int mg_subiso_batch_count_orders(void* dgraph, const mg_csr_view* const* qs, uint32_t nq,
                                 const uint32_t* orders, const mg_opts* opts, uint64_t* counts,
                                 uint64_t* level_rows, mg_stats* st) {
  MG_ENTRY(dgraph);
  if (!qs || !counts || nq == 0) return mg::set_error(MG_E_ARG, "null argument or empty batch");
  try {
    return mg::subiso_batch(dg, qs, nq, opts, counts, st, orders, level_rows);
  } catch (const std::bad_alloc&) {
    return mg::set_error(MG_E_OOM, "host allocation failed");
  }
}

int mg_plan_orders(void* dgraph, const mg_csr_view* const* qs, uint32_t nq, const mg_opts* opts,
                   uint32_t* orders) {
  MG_ENTRY(dgraph);
  if (!qs || !orders || nq == 0) return mg::set_error(MG_E_ARG, "null argument or empty batch");
  try {
    const mg_opts o = mg::resolve_opts(opts);
    std::vector<mg::QueryGraph> Q(nq);
    for (uint32_t i = 0; i < nq; ++i) {
      int rc = mg::normalise_query(qs[i], &Q[i]);
      if (rc) return mg::set_error(rc, "query %u: %s", i, mg::last_error_cstr());
    }
    std::memset(orders, 0, uint64_t(nq) * MG_MAX_QUERY_VERTICES * 4);
    if (o.order == MG_ORDER_LEARNED && o.model) {
      int rc = mg::ensure_full_stats(dg);
      if (rc) return rc;
      std::vector<const mg::QueryGraph*> qp(nq);
      for (uint32_t i = 0; i < nq; ++i) qp[i] = &Q[i];
      std::vector<std::array<uint32_t, MG_MAX_QUERY_VERTICES>> ord;
      if ((rc = mg::order_learned_batch(o.model, qp, dg->stats, ord))) return rc;
      for (uint32_t i = 0; i < nq; ++i)
        std::memcpy(orders + uint64_t(i) * MG_MAX_QUERY_VERTICES, ord[i].data(), Q[i].k * 4);
      return MG_OK;
    }
    for (uint32_t i = 0; i < nq; ++i) {
      int rc = mg::choose_order(dg, Q[i], o, orders + uint64_t(i) * MG_MAX_QUERY_VERTICES);
      if (rc) return rc;
    }
    return MG_OK;
  } catch (const std::bad_alloc&) {
    return mg::set_error(MG_E_OOM, "host allocation failed");
  }
}

int mg_selftest_wait_timeout(void* dgraph, const mg_csr_view* q, uint32_t spin_limit,
                             int* status) {
  MG_ENTRY(dgraph);
  if (!q || !status || spin_limit == 0) return mg::set_error(MG_E_ARG, "bad argument");
  uint64_t err = 0;
  int rc = mg::selftest_wait(dg, q, spin_limit, &err);
  if (rc) return rc;
  *status = (err & mg::ERR_TIMEOUT) ? MG_E_TIMEOUT : MG_OK;
  return MG_OK;
}

}  // extern "C"

// ---------------------------------------------------------------------------
// Allocation-free count (mg_subiso_count_noalloc)
//
// For callers that cannot allocate device memory when they ask for a count:
// processes whose device memory is owned by another allocator (a framework's
// caching allocator that has reserved nearly all HBM, a fixed arena), or
// latency-critical paths that must not pay cudaMalloc/cudaFree and the
// device-wide synchronisation cudaFree implies.  The level tables, scan
// scratch, counters and the plan live in the file-scope array below, sized
// once at load time and held by every GPU that loads the library until the
// process exits.  The data graph must already be resident (mg_graph_upload).
// ---------------------------------------------------------------------------
namespace mg {

static __device__ __align__(256) unsigned char g_noalloc_scratch[MG_NOALLOC_SCRATCH_BYTES];

namespace {

// Device address of g_noalloc_scratch per device, looked up once per device
// (with that device current) by the first call on it.
std::mutex g_noalloc_mu;  // one call at a time: every call shares the array
void* g_noalloc_ptr[256] = {};

int noalloc_scratch(int device, unsigned char** out) {
  if (device < 0 || device >= 256) return set_error(MG_E_ARG, "device %d out of range", device);
  if (!g_noalloc_ptr[device]) {
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess || !p)
      return set_error(MG_E_CUDA, "cudaGetSymbolAddress(g_noalloc_scratch) on device %d: %s",
                       device, cudaGetErrorString(e));
    g_noalloc_ptr[device] = p;
  }
  *out = static_cast<unsigned char*>(g_noalloc_ptr[device]);
  return MG_OK;
}

// Level tables of a single-query count, carved out of `base`.
struct NoallocLayout {
  unsigned long long* res;
  PlanDev* plan;
  unsigned long long* status;
  uint32_t* tile_row;
  uint32_t* col[MAXK][MAXK];
  uint64_t* woff[MAXK];
  uint32_t* dstart[MAXK];
  uint8_t* dci[MAXK];
};

// Elements per expand launch of a level whose survivors are not stored.
constexpr uint64_t kNoallocSegment = 1ull << 24;

// Look-back words of tables of `cap` rows (a single vertex needs none).
uint64_t noalloc_status_bytes(uint64_t cap, uint32_t k) {
  return (k > 1 ? cap / WS_ROWS + 2 : 1) * 8;
}

// Bytes that tables of `cap` rows are charged with.  A fixed formula that
// bounds the layout below, so that the chunk_rows that fit the scratch do not
// change with it.
uint64_t noalloc_charge(uint64_t cap, uint32_t k) {
  uint64_t off = 0;
  auto take = [&](uint64_t bytes) { off = ((off + 255) & ~uint64_t(255)) + bytes; };
  for (uint64_t bytes : {uint64_t(72 * 8), uint64_t(8), uint64_t((MAXK + 1) * 8),
                         uint64_t(sizeof(PlanDev)), (cap / 4096 + 2) * 8,
                         (kNoallocSegment / 256 + 2) * 4})
    take(bytes);
  for (uint32_t l = 0; l < k; ++l) {
    const uint64_t rows = l == 0 ? 1 : cap;
    for (uint32_t j = 0; j <= l; ++j) take(rows * 4);
    take((rows + 1) * 8);
    take(rows * 4);
    take(rows);
  }
  return off;
}

uint64_t noalloc_carve(unsigned char* base, uint64_t cap, uint32_t k, NoallocLayout* L) {
  uint64_t off = 0;
  auto take = [&](uint64_t bytes) -> unsigned char* {
    off = (off + 255) & ~uint64_t(255);
    unsigned char* p = base + off;
    off += bytes;
    return p;
  };
  L->res = reinterpret_cast<unsigned long long*>(take(res_words(1) * 8));
  L->plan = reinterpret_cast<PlanDev*>(take(sizeof(PlanDev)));
  L->status = reinterpret_cast<unsigned long long*>(take(noalloc_status_bytes(cap, k)));
  L->tile_row = reinterpret_cast<uint32_t*>(take((kNoallocSegment / EXPAND_TILE + 2) * 4));
  for (uint32_t l = 0; l < k; ++l) {
    const uint64_t rows = l == 0 ? 1 : cap;
    for (uint32_t j = 0; j < l; ++j) L->col[l][j] = reinterpret_cast<uint32_t*>(take(rows * 4));
    L->woff[l] = reinterpret_cast<uint64_t*>(take((rows + 1) * 8));
    L->dstart[l] = reinterpret_cast<uint32_t*>(take(rows * 4));
    L->dci[l] = reinterpret_cast<uint8_t*>(take(rows));
  }
  return off;
}

int noalloc_count(DevGraph* dg, const mg_csr_view* q, const mg_opts* opts, uint64_t* count) {
  mg_opts o;
  mg_opts_default(&o);
  if (opts) o = *opts;
  // Every argument is checked before any work is queued on the shared array.
  int rc = check_opts(o);
  if (rc) return rc;
  if (o.matrix_filter)
    return set_error(MG_E_ARG, "mg_subiso_count_noalloc does not apply a matrix filter");
  QueryGraph Q;
  rc = normalise_query(q, &Q);  // the allocating entry points' normaliser
  if (rc) return rc;
  uint32_t order[MAXK];
  if (o.order == MG_ORDER_REFERENCE) {
    order_reference(Q, order);
  } else if (o.order == MG_ORDER_STRONG) {
    order_strong(Q, dg->stats, order);
  } else if (o.order == MG_ORDER_GIVEN) {
    if (!o.given_order) return set_error(MG_E_ARG, "MG_ORDER_GIVEN without given_order");
    std::memcpy(order, o.given_order, Q.k * 4);
    if (!order_is_permutation(order, Q.k))
      return set_error(MG_E_ARG, "given_order is not a permutation of 0..%u", Q.k - 1);
  } else {
    return set_error(MG_E_ARG, "mg_subiso_count_noalloc supports the reference, strong and "
                               "given orders only");
  }
  PlanDev P;
  if ((rc = build_plan(dg, Q, order, &P))) return rc;
  const uint32_t k = P.k;

  // Rows per level table: the largest power of two whose layout fits, or the
  // caller's chunk_rows, which must fit.
  NoallocLayout L;
  uint64_t cap = 0;
  if (o.chunk_rows) {
    if (o.chunk_rows > (1ull << 31) ||
        noalloc_charge(o.chunk_rows, k) > MG_NOALLOC_SCRATCH_BYTES)
      return set_error(MG_E_LIMIT,
                       "chunk_rows=%llu for a %u-vertex query needs %llu bytes of scratch; the "
                       "static scratch holds %llu bytes",
                       (unsigned long long)o.chunk_rows, k,
                       (unsigned long long)noalloc_charge(
                           std::min<uint64_t>(o.chunk_rows, 1ull << 31), k),
                       (unsigned long long)MG_NOALLOC_SCRATCH_BYTES);
    cap = o.chunk_rows;
  } else {
    for (uint64_t c = 1ull << 22; c >= 64; c >>= 1)
      if (noalloc_charge(c, k) <= MG_NOALLOC_SCRATCH_BYTES) {
        cap = c;
        break;
      }
    if (!cap)
      return set_error(MG_E_LIMIT, "a %u-vertex query does not fit the %llu-byte static scratch",
                       k, (unsigned long long)MG_NOALLOC_SCRATCH_BYTES);
  }
  unsigned char* base = nullptr;
  if ((rc = noalloc_scratch(dg->device, &base))) return rc;
  if (noalloc_carve(base, cap, k, &L) > MG_NOALLOC_SCRATCH_BYTES)
    return set_error(MG_E_LIMIT, "tables of %llu rows do not fit the static scratch",
                     (unsigned long long)cap);

  cudaStream_t st = dg->stream;
  // The array keeps the previous call's contents: counters start at zero.
  MG_CK(cudaMemcpyAsync(L.plan, &P, sizeof(PlanDev), cudaMemcpyHostToDevice, st));
  MG_CK(cudaMemsetAsync(L.res, 0, res_words(1) * 8, st));
  MG_CK(cudaMemsetAsync(L.status, 0, noalloc_status_bytes(cap, k), st));

  StepArgs a;
  std::memset(&a, 0, sizeof(a));
  a.g = dg->g;
  a.plans = L.plan;
  a.count_mode = 1;
  a.filters = o.filters & MG_FILTER_ALL;
  a.nq = 1;
  a.grab = o.grab;
  a.root_step = o.root_step > 1 ? o.root_step : 1u;
  a.probe_min = o.probe_min ? o.probe_min : kProbeMin;
  if (o.root_end || a.root_step > 1) {
    a.root_begin = o.root_begin;
    a.root_end = o.root_end ? o.root_end : ~0ull;
  }
  unsigned long long h[res_words(1)];
  uint32_t epoch = 0;
  WalkBufs B;
  B.cap = cap;
  B.col = L.col;
  B.woff = L.woff;
  B.dstart = L.dstart;
  B.dci = L.dci;
  B.tile_row = L.tile_row;
  B.seg = kNoallocSegment;
  B.status = L.status;
  B.status_bytes = noalloc_status_bytes(cap, k);
  B.epoch = &epoch;
  B.res = L.res;
  B.h_res = h;
  RunResult res;
  o.kernel_events = 0;
  if ((rc = walk_levels(dg, &P, 1, true, o, a, B, &res))) {
    cudaStreamSynchronize(st);  // nothing of this call stays queued on the array
    return rc;
  }
  *count = h[C_NUM];
  return MG_OK;
}

}  // namespace
}  // namespace mg

extern "C" int mg_subiso_count_noalloc(void* dgraph, const mg_csr_view* q, const mg_opts* opts,
                                       uint64_t* count) {
  mg::clear_error();
  if (!dgraph || !q || !count) return mg::set_error(MG_E_ARG, "null argument");
  auto* dg = static_cast<mg::DevGraph*>(dgraph);
  std::lock_guard<std::mutex> glock(mg::g_noalloc_mu);
  std::lock_guard<std::mutex> lock(dg->mu);
  mg::DeviceGuard guard(dg->device);
  return mg::noalloc_count(dg, q, opts, count);
}
