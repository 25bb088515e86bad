// Data-graph upload and the derived device indices.
//
// The reference keeps the raw CSR byte buffer in managed memory and
// re-derives labels and degrees inside every filter call
// (core/task/gpu_task/kernel/kernel_woj_subsio.cu:545-561, :753-815).  Here
// the graph is uploaded once into plain device memory and turned into
// label-sliced adjacency (each list reordered by (label, id)), neighbour-label
// bit words (the sound subset form of NeighborLabelCounterFilter,
// kernel_woj_subsio.cu:385-446) and label buckets (the level-0 candidate
// ranges).
#include <algorithm>
#include <functional>
#include <cstdlib>
#include <cstring>
#include <thread>

#include <cub/cub.cuh>

#include "mg_device.cuh"

namespace mg {

int dev_alloc(DevGraph* dg, void** p, size_t bytes) {
  *p = nullptr;
  if (bytes == 0) bytes = 16;
  cudaError_t e = cudaMalloc(p, bytes);
  if (e != cudaSuccess) {
    cudaGetLastError();
    *p = nullptr;
    return set_error(MG_E_OOM, "cudaMalloc(%zu) failed: %s", bytes, cudaGetErrorString(e));
  }
  dg->allocs.push_back(*p);
  dg->info.device_bytes += bytes;
  return MG_OK;
}

void free_workspace(Workspace* ws);
void free_lanes(LaneSet* ls);

DevGraph::~DevGraph() {
  if (stream) {
    int prev = 0;
    cudaGetDevice(&prev);
    cudaSetDevice(device);
    cudaStreamSynchronize(stream);
    free_workspace(ws);
    free_lanes(lanes);
    cudaFree(emit_mem);
    for (void* p : allocs) cudaFree(p);
    cudaStreamDestroy(stream);
    cudaSetDevice(prev);
  }
}

namespace {

// Global -> local id through a dense table over [0, max_vid].
__global__ void k_build_g2l(const uint32_t* globalid, uint32_t n, uint32_t* g2l,
                            uint32_t max_vid, uint32_t* err) {
  for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < n;
       i += uint64_t(gridDim.x) * blockDim.x) {
    uint32_t gid = globalid[i];
    if (gid > max_vid) {
      atomicOr(err, ERR_RANGE);
      continue;
    }
    g2l[gid] = uint32_t(i);
  }
}

__global__ void k_map_edges(uint32_t* adj, uint64_t m, const uint32_t* g2l,
                            uint32_t max_vid, uint32_t* err) {
  for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < m;
       i += uint64_t(gridDim.x) * blockDim.x) {
    uint32_t gid = adj[i];
    uint32_t l = gid <= max_vid ? g2l[gid] : FULL;
    if (l == FULL) atomicOr(err, ERR_RANGE);
    adj[i] = l == FULL ? 0 : l;
  }
}

// Warp per vertex: flags unsorted or repeated entries and ids >= n.
__global__ void k_check_lists(const uint32_t* off, const uint32_t* adj, uint32_t n,
                              uint32_t* flags) {
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t warp = (blockIdx.x * uint64_t(blockDim.x) + threadIdx.x) >> 5;
  const uint64_t nwarps = (uint64_t(gridDim.x) * blockDim.x) >> 5;
  uint32_t bad = 0;
  for (uint64_t v = warp; v < n; v += nwarps) {
    const uint32_t s = off[v], e = off[v + 1];
    for (uint32_t j = s + lane; j < e; j += 32) {
      uint32_t a = adj[j];
      if (a >= n) bad |= 2;
      if (j + 1 < e && a >= adj[j + 1]) bad |= 1;
    }
  }
  bad = __reduce_or_sync(FULL, bad);
  if (lane == 0 && bad) atomicOr(flags, bad);
}

// Distinct entries per (sorted) list.
__global__ void k_count_unique(const uint32_t* off, const uint32_t* adj, uint32_t n,
                               uint32_t* newdeg) {
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t warp = (blockIdx.x * uint64_t(blockDim.x) + threadIdx.x) >> 5;
  const uint64_t nwarps = (uint64_t(gridDim.x) * blockDim.x) >> 5;
  for (uint64_t v = warp; v < n; v += nwarps) {
    const uint32_t s = off[v], e = off[v + 1];
    uint32_t c = 0;
    for (uint32_t j = s + lane; j < e; j += 32) c += (j == s || adj[j] != adj[j - 1]);
    c = __reduce_add_sync(FULL, c);
    if (lane == 0) newdeg[v] = c;
  }
}

__global__ void k_compact_unique(const uint32_t* off, const uint32_t* adj, uint32_t n,
                                 const uint32_t* newoff, uint32_t* out) {
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t warp = (blockIdx.x * uint64_t(blockDim.x) + threadIdx.x) >> 5;
  const uint64_t nwarps = (uint64_t(gridDim.x) * blockDim.x) >> 5;
  for (uint64_t v = warp; v < n; v += nwarps) {
    const uint32_t s = off[v], e = off[v + 1];
    uint32_t base = newoff[v];
    for (uint32_t j0 = s; j0 < e; j0 += 32) {
      uint32_t j = j0 + lane;
      bool keep = j < e && (j == s || adj[j] != adj[j - 1]);
      uint32_t bal = __ballot_sync(FULL, keep);
      if (keep) out[base + __popc(bal & ((1u << lane) - 1))] = adj[j];
      base += __popc(bal);
    }
  }
}

// ---- label-sliced adjacency --------------------------------------------------
// The lists (off, adj: input ids) become one CSR per neighbour label over the
// vertices in their label order:
//   k_label_count    entries of every (label, vertex), into loff;
//   scan             loff becomes slice starts (exclusive prefix sums);
//   k_label_scatter  every entry to its slice, in list order (stable).
// A block takes PT_V consecutive vertices and keeps its counts or cursors of
// all labels in shared memory, so that loff is read and written in rows of
// consecutive vertices and the slices a block writes lie side by side.  A
// list longer than PT_LONG is walked by the whole block: hubs come first in
// every label bucket of an unpermuted power-law graph.
constexpr int PT_BLOCK = 256, PT_WARPS = PT_BLOCK / 32;
constexpr int PT_V = 32, PT_STRIDE = PT_V + 1;
constexpr uint32_t PT_LONG = 1024;

__global__ void __launch_bounds__(PT_BLOCK) k_label_count(
    const uint32_t* __restrict__ off, const uint32_t* __restrict__ adj, uint32_t n,
    const uint32_t* __restrict__ input_id, const uint8_t* __restrict__ label, uint32_t L,
    uint32_t W, uint32_t* loff, uint32_t* nlb, uint32_t* deg, uint32_t* selfbits) {
  extern __shared__ uint32_t hist[];  // [L][PT_STRIDE]
  __shared__ uint32_t self;           // one word: PT_V vertices
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (uint32_t x = threadIdx.x; x < L * PT_STRIDE; x += PT_BLOCK) hist[x] = 0;
  if (threadIdx.x == 0) self = 0;
  __syncthreads();
  const uint32_t v0 = blockIdx.x * PT_V;
  auto walk = [&](uint32_t j, uint32_t s, uint32_t e, uint32_t v, uint32_t at, uint32_t step) {
    bool me = false;
    for (uint32_t x = s + at; x < e; x += step) {
      const uint32_t u = __ldg(adj + x);
      me |= u == v;
      atomicAdd(&hist[label[u] * PT_STRIDE + j], 1u);
    }
    if (me) atomicOr(&self, 1u << j);
  };
  for (uint32_t j = warp; j < PT_V && v0 + j < n; j += PT_WARPS) {
    const uint32_t v = input_id[v0 + j], s = off[v], e = off[v + 1];
    if (lane == 0) deg[v0 + j] = e - s;
    if (e - s <= PT_LONG) walk(j, s, e, v, lane, 32);
  }
  for (uint32_t j = 0; j < PT_V && v0 + j < n; ++j) {
    const uint32_t v = input_id[v0 + j], s = off[v], e = off[v + 1];
    if (e - s > PT_LONG) walk(j, s, e, v, threadIdx.x, PT_BLOCK);
  }
  __syncthreads();
  const uint32_t nv = min(uint32_t(PT_V), n - v0);
  if (lane < nv)
    for (uint32_t l = warp; l < L; l += PT_WARPS)
      loff[uint64_t(l) * n + v0 + lane] = hist[l * PT_STRIDE + lane];
  for (uint32_t j = warp; j < nv; j += PT_WARPS)
    for (uint32_t w = 0; w < W; ++w) {
      const uint32_t l = w * 32 + lane;
      const uint32_t bits = __ballot_sync(FULL, l < L && hist[l * PT_STRIDE + j] > 0);
      if (lane == 0) nlb[uint64_t(v0 + j) * W + w] = bits;
    }
  if (threadIdx.x == 0) selfbits[v0 >> 5] |= self;  // PT_V == 32: this block's word
}

__global__ void __launch_bounds__(PT_BLOCK) k_label_scatter(
    const uint32_t* __restrict__ off, const uint32_t* __restrict__ adj, uint32_t n,
    const uint32_t* __restrict__ input_id, const uint32_t* __restrict__ new_id,
    const uint8_t* __restrict__ label, uint32_t L, const uint32_t* __restrict__ loff,
    uint32_t* out) {
  extern __shared__ uint32_t sh[];
  uint32_t* cur = sh;                       // [L][PT_STRIDE] next position of every slice
  uint32_t* part = sh + L * PT_STRIDE;      // [PT_WARPS][L] a long list's parts
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t v0 = blockIdx.x * PT_V;
  const uint32_t nv = min(uint32_t(PT_V), n - v0);
  if (lane < nv)
    for (uint32_t l = warp; l < L; l += PT_WARPS)
      cur[l * PT_STRIDE + lane] = loff[uint64_t(l) * n + v0 + lane];
  __syncthreads();
  // Entries [s, e) in order by one warp; at[l * stride] is the next position of
  // label l.
  auto place = [&](uint32_t s, uint32_t e, uint32_t* at, uint32_t stride) {
    for (uint32_t x0 = s; x0 < e; x0 += 32) {
      const bool valid = x0 + lane < e;
      const uint32_t u = valid ? __ldg(adj + x0 + lane) : 0u;
      const uint32_t l = valid ? label[u] : FULL;
      const uint32_t id = valid ? __ldg(new_id + u) : 0u;
      const uint32_t peers = __match_any_sync(FULL, l);
      const uint32_t rank = __popc(peers & ((1u << lane) - 1));
      const uint32_t base = valid ? at[l * stride] : 0u;
      __syncwarp();
      if (valid) {
        out[base + rank] = id;
        if (rank == 0) at[l * stride] = base + __popc(peers);
      }
      __syncwarp();
    }
  };
  for (uint32_t j = warp; j < nv; j += PT_WARPS) {
    const uint32_t v = input_id[v0 + j], s = off[v], e = off[v + 1];
    if (e - s <= PT_LONG) place(s, e, cur + j, PT_STRIDE);
  }
  for (uint32_t j = 0; j < nv; ++j) {
    const uint32_t v = input_id[v0 + j], s = off[v], e = off[v + 1];
    if (e - s <= PT_LONG) continue;
    // every warp a consecutive part: count it, then place it behind the parts
    // before it
    const uint32_t per = (e - s + PT_WARPS - 1) / PT_WARPS;
    const uint32_t ws = min(e, s + warp * per), we = min(e, ws + per);
    uint32_t* mine = part + warp * L;
    for (uint32_t l = lane; l < L; l += 32) mine[l] = 0;
    __syncwarp();
    for (uint32_t x = ws + lane; x < we; x += 32) atomicAdd(&mine[label[__ldg(adj + x)]], 1u);
    __syncthreads();
    for (uint32_t l = threadIdx.x; l < L; l += PT_BLOCK) {
      uint32_t at = cur[l * PT_STRIDE + j];
      for (uint32_t w = 0; w < PT_WARPS; ++w) {
        const uint32_t c = part[w * L + l];
        part[w * L + l] = at;
        at += c;
      }
    }
    __syncthreads();
    place(ws, we, mine, 1);
    __syncthreads();
  }
}

// Exclusive prefix sums of N 32-bit words in place (sums below 2^32), the total
// to p[N]: sums of tiles, their prefix sums, then every tile on its own.
constexpr int SC_BLOCK = 256, SC_PER = 32, SC_TILE = SC_BLOCK * SC_PER;

__device__ __forceinline__ uint32_t warp_incl(uint32_t v) {
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t t = __shfl_up_sync(FULL, v, d);
    if ((threadIdx.x & 31) >= d) v += t;
  }
  return v;
}

// Exclusive prefix of v over the block; *total is the block's sum.
__device__ __forceinline__ uint32_t block_excl(uint32_t v, uint32_t* total) {
  __shared__ uint32_t ws[33];
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const uint32_t incl = warp_incl(v);
  if (lane == 31) ws[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    const uint32_t s = lane < nw ? ws[lane] : 0u, si = warp_incl(s);
    __syncwarp();
    if (lane < nw) ws[lane] = si - s;
    if (lane == 31) ws[32] = si;
  }
  __syncthreads();
  const uint32_t res = ws[warp] + incl - v;
  *total = ws[32];
  __syncthreads();
  return res;
}

__global__ void __launch_bounds__(SC_BLOCK) k_sum_tiles(const uint32_t* __restrict__ p, uint64_t N,
                                                        uint32_t* sums) {
  const uint64_t base = uint64_t(blockIdx.x) * SC_TILE;
  uint32_t s = 0;
  for (uint32_t j = threadIdx.x; j < SC_TILE; j += SC_BLOCK)
    if (base + j < N) s += p[base + j];
  uint32_t total;
  block_excl(s, &total);
  if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

__global__ void __launch_bounds__(1024) k_scan_sums(uint32_t* sums, uint32_t nb, uint32_t* total) {
  uint32_t carry = 0;
  for (uint32_t b = 0; b < nb; b += 1024 * 8) {
    uint32_t v[8], s = 0, t;
    const uint32_t at = b + threadIdx.x * 8;
    for (int j = 0; j < 8; ++j) s += v[j] = at + j < nb ? sums[at + j] : 0u;
    uint32_t ex = carry + block_excl(s, &t);
    for (int j = 0; j < 8; ++j) {
      if (at + j < nb) sums[at + j] = ex;
      ex += v[j];
    }
    carry += t;
  }
  if (threadIdx.x == 0) *total = carry;
}

__global__ void __launch_bounds__(SC_BLOCK) k_scan_tiles(uint32_t* p, uint64_t N,
                                                         const uint32_t* __restrict__ sums) {
  __shared__ uint32_t tile[SC_TILE + SC_TILE / 32];
  const uint64_t base = uint64_t(blockIdx.x) * SC_TILE;
  for (uint32_t j = threadIdx.x; j < SC_TILE; j += SC_BLOCK)
    tile[j + (j >> 5)] = base + j < N ? p[base + j] : 0u;
  __syncthreads();
  const uint32_t at = threadIdx.x * (SC_PER + 1);
  uint32_t s = 0, t;
  for (int j = 0; j < SC_PER; ++j) s += tile[at + j];
  uint32_t ex = sums[blockIdx.x] + block_excl(s, &t);
  for (int j = 0; j < SC_PER; ++j) {
    const uint32_t v = tile[at + j];
    tile[at + j] = ex;
    ex += v;
  }
  __syncthreads();
  for (uint32_t j = threadIdx.x; j < SC_TILE; j += SC_BLOCK)
    if (base + j < N) p[base + j] = tile[j + (j >> 5)];
}

__global__ void k_set_u32(uint32_t* p, uint64_t i, uint32_t v) { p[i] = v; }

// globalid of every vertex from the global ids in input order.
__global__ void k_permute_u32(const uint32_t* __restrict__ src, const uint32_t* __restrict__ idx,
                              uint32_t n, uint32_t* dst) {
  for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < n;
       i += uint64_t(gridDim.x) * blockDim.x)
    dst[i] = src[idx[i]];
}

// Per-label degree sums / maxima / log2 histograms and label-pair edge counts
// (features of the order model): a block per (label bucket part), a neighbour
// label at a time over consecutive vertices.
constexpr uint32_t LS_PART = 8192;  // vertices per block
__global__ void __launch_bounds__(256) k_label_stats(
    const uint32_t* __restrict__ loff, const uint32_t* __restrict__ deg,
    const uint32_t* __restrict__ bucket_off, uint32_t n, uint32_t L,
    unsigned long long* deg_sum, unsigned int* deg_max, unsigned long long* deg_hist,
    unsigned long long* pair) {
  const uint32_t lv = blockIdx.y, lane = threadIdx.x & 31;
  const uint32_t b0 = bucket_off[lv], b1 = bucket_off[lv + 1];
  __shared__ unsigned long long hist[33];
  for (uint64_t v0 = b0 + uint64_t(blockIdx.x) * LS_PART; v0 < b1;
       v0 += uint64_t(gridDim.x) * LS_PART) {
    const uint32_t v1 = uint32_t(min(v0 + LS_PART, uint64_t(b1)));
    if (threadIdx.x < 33) hist[threadIdx.x] = 0;
    __syncthreads();
    unsigned long long sum = 0;
    uint32_t mx = 0;
    for (uint32_t v = uint32_t(v0) + threadIdx.x; v < v1; v += blockDim.x) {
      const uint32_t d = deg[v];
      sum += d;
      mx = max(mx, d);
      atomicAdd(&hist[d == 0 ? 0 : 32 - __clz(d)], 1ull);
    }
    for (int d = 16; d > 0; d >>= 1) sum += __shfl_down_sync(FULL, sum, d);
    mx = __reduce_max_sync(FULL, mx);
    if (lane == 0) {
      atomicAdd(&deg_sum[lv], sum);
      atomicMax(&deg_max[lv], mx);
    }
    __syncthreads();
    if (threadIdx.x < 33 && hist[threadIdx.x])
      atomicAdd(&deg_hist[lv * 33 + threadIdx.x], hist[threadIdx.x]);
    __syncthreads();
    // the entries of consecutive vertices to one label are one range of adj
    for (uint32_t l = threadIdx.x; l < L; l += blockDim.x) {
      const uint32_t c = loff[uint64_t(l) * n + v1] - loff[uint64_t(l) * n + v0];
      if (c) atomicAdd(&pair[lv * uint64_t(L) + l], (unsigned long long)c);
    }
  }
}

unsigned host_threads() {
  unsigned t = std::thread::hardware_concurrency();
  return t == 0 ? 1 : std::min(t, 32u);
}

bool arrays_equal(const uint32_t* a, const uint32_t* b, uint64_t words) {
  if (a == b) return true;
  unsigned T = host_threads();
  if (words < (1u << 20)) T = 1;
  std::vector<std::thread> ts;
  std::vector<char> eq(T, 1);
  uint64_t chunk = (words + T - 1) / T;
  for (unsigned t = 0; t < T; ++t)
    ts.emplace_back([&, t]() {
      uint64_t lo = t * chunk, hi = std::min(words, lo + chunk);
      if (lo < hi) eq[t] = std::memcmp(a + lo, b + lo, (hi - lo) * 4) == 0;
    });
  for (auto& th : ts) th.join();
  for (char c : eq)
    if (!c) return false;
  return true;
}

inline unsigned grid_for(uint64_t items, unsigned block, unsigned cap) {
  uint64_t g = (items + block - 1) / block;
  return unsigned(std::max<uint64_t>(1, std::min<uint64_t>(g, cap)));
}

}  // namespace

// Hub bitmaps: block h sets the bits of hub h's whole d-adjacency, a label
// slice per warp at a time.
__global__ void __launch_bounds__(256) k_hub_bits(const uint32_t* __restrict__ adj,
                                                  const uint32_t* __restrict__ loff, uint32_t n,
                                                  uint32_t L, const uint32_t* __restrict__ hub_vid,
                                                  uint32_t words, uint32_t* bits) {
  const uint32_t y = hub_vid[blockIdx.x];
  uint32_t* row = bits + uint64_t(blockIdx.x) * words;
  for (uint32_t l = threadIdx.x >> 5; l < L; l += blockDim.x >> 5) {
    const uint32_t s = loff[uint64_t(l) * n + y], e = loff[uint64_t(l) * n + y + 1];
    for (uint32_t j = s + (threadIdx.x & 31); j < e; j += 32) {
      const uint32_t x = adj[j];
      atomicOr(row + (x >> 5), 1u << (x & 31));
    }
  }
}

// Selects the hubs of direction d (decreasing degree within the byte budget,
// ties at the cut all in or all out) and builds their bitmaps.
static int build_hubs(DevGraph* dg, int d, const std::vector<uint32_t>& deg, uint64_t budget,
                      uint32_t min_degree) {
  const uint32_t n = dg->g.n;
  const uint32_t words = ((n + 31) / 32 + 3) & ~3u;  // rows start on 16-byte boundaries
  const uint64_t row_bytes = uint64_t(words) * 4;
  uint64_t cap = std::min<uint64_t>(budget / row_bytes, NO_HUB);
  if (cap == 0) return MG_OK;
  std::vector<uint32_t> cand;
  for (uint32_t v = 0; v < n; ++v)
    if (deg[v] >= min_degree) cand.push_back(v);
  if (cand.empty()) return MG_OK;
  uint32_t cut = min_degree;
  if (cand.size() > cap) {
    std::vector<uint32_t> dv(cand.size());
    for (size_t i = 0; i < cand.size(); ++i) dv[i] = deg[cand[i]];
    std::nth_element(dv.begin(), dv.begin() + (cap - 1), dv.end(), std::greater<uint32_t>());
    cut = dv[cap - 1];  // the cap-th largest degree
    uint64_t at_or_above = 0;
    for (uint32_t x : dv) at_or_above += x >= cut;
    if (at_or_above > cap) ++cut;  // ties at the cut would overflow: leave them out
  }
  std::vector<uint32_t> hub_vid;
  std::vector<uint16_t> slot(n, NO_HUB);
  for (uint32_t v : cand)
    if (deg[v] >= cut) {
      slot[v] = uint16_t(hub_vid.size());
      hub_vid.push_back(v);
    }
  if (hub_vid.empty()) return MG_OK;
  cudaStream_t st = dg->stream;
  uint16_t* d_slot;
  uint32_t* d_bits;  // the rows, and behind them the vertices they are built from
  int rc;
  if ((rc = dev_alloc(dg, (void**)&d_slot, uint64_t(n) * 2))) return rc;
  if ((rc = dev_alloc(dg, (void**)&d_bits, hub_vid.size() * (row_bytes + 4)))) return rc;
  uint32_t* d_vid = d_bits + hub_vid.size() * words;
  MG_CK(cudaMemcpyAsync(d_slot, slot.data(), uint64_t(n) * 2, cudaMemcpyHostToDevice, st));
  MG_CK(cudaMemcpyAsync(d_vid, hub_vid.data(), hub_vid.size() * 4, cudaMemcpyHostToDevice, st));
  MG_CK(cudaMemsetAsync(d_bits, 0, hub_vid.size() * row_bytes, st));
  k_hub_bits<<<unsigned(hub_vid.size()), 256, 0, st>>>(dg->g.adj[d], dg->g.loff[d], n, dg->g.L,
                                                      d_vid, words, d_bits);
  MG_CK(cudaGetLastError());
  MG_CK(cudaStreamSynchronize(st));
  dg->g.hub_slot[d] = d_slot;
  dg->g.hub_bits[d] = d_bits;
  dg->g.hub_words = words;
  dg->info.hubs += uint32_t(hub_vid.size());
  dg->info.hub_min_degree = cut;
  dg->info.hub_bytes += hub_vid.size() * row_bytes;
  return MG_OK;
}

// Builds adjacency + slices for one direction from raw host arrays.
static int build_direction(DevGraph* dg, int d, const uint32_t* h_off, const uint32_t* h_adj,
                           uint32_t m, const uint32_t* d_g2l, uint32_t max_vid,
                           const uint32_t* d_new, const uint8_t* d_label, uint32_t* d_err) {
  cudaStream_t st = dg->stream;
  const uint32_t n = dg->g.n, L = dg->g.L, W = dg->g.W;
  uint32_t *off = nullptr, *adj = nullptr;
  MG_CK(cudaMallocAsync((void**)&off, (uint64_t(n) + 1) * 4, st));
  MG_CK(cudaMallocAsync((void**)&adj, std::max<uint64_t>(1, m) * 4ull, st));
  MG_CK(cudaMemcpyAsync(off, h_off, (uint64_t(n) + 1) * 4, cudaMemcpyHostToDevice, st));
  if (m) MG_CK(cudaMemcpyAsync(adj, h_adj, uint64_t(m) * 4, cudaMemcpyHostToDevice, st));
  if (d_g2l && m) k_map_edges<<<grid_for(m, 256, dg->sms * 32), 256, 0, st>>>(adj, m, d_g2l, max_vid, d_err);
  uint32_t* d_flags = d_err + 1;
  MG_CK(cudaMemsetAsync(d_flags, 0, 4, st));
  k_check_lists<<<grid_for(uint64_t(n) * 32, 256, dg->sms * 32), 256, 0, st>>>(off, adj, n, d_flags);
  uint32_t flags = 0;
  MG_CK(cudaMemcpyAsync(&flags, d_flags, 4, cudaMemcpyDeviceToHost, st));
  MG_CK(cudaStreamSynchronize(st));
  if (flags & 2) {
    cudaFreeAsync(off, st);
    cudaFreeAsync(adj, st);
    return set_error(MG_E_FORMAT, "adjacency entry outside the vertex range");
  }
  uint32_t mm = m;
  if (flags & 1) {
    // Unsorted or repeated entries: segmented sort, then drop repeats.
    uint32_t* sorted = nullptr;
    MG_CK(cudaMallocAsync((void**)&sorted, std::max<uint64_t>(1, m) * 4ull, st));
    size_t tmp_bytes = 0;
    MG_CK(cub::DeviceSegmentedSort::SortKeys(nullptr, tmp_bytes, adj, sorted, m, n, off,
                                             off + 1, st));
    void* tmp = nullptr;
    MG_CK(cudaMallocAsync(&tmp, std::max<size_t>(16, tmp_bytes), st));
    MG_CK(cub::DeviceSegmentedSort::SortKeys(tmp, tmp_bytes, adj, sorted, m, n, off,
                                             off + 1, st));
    cudaFreeAsync(tmp, st);
    uint32_t *newdeg = nullptr, *newoff = nullptr;
    MG_CK(cudaMallocAsync((void**)&newdeg, (uint64_t(n) + 1) * 4, st));
    MG_CK(cudaMallocAsync((void**)&newoff, (uint64_t(n) + 1) * 4, st));
    k_count_unique<<<grid_for(uint64_t(n) * 32, 256, dg->sms * 32), 256, 0, st>>>(off, sorted, n, newdeg);
    tmp_bytes = 0;
    MG_CK(cub::DeviceScan::ExclusiveSum(nullptr, tmp_bytes, newdeg, newoff, n + 1, st));
    MG_CK(cudaMallocAsync(&tmp, std::max<size_t>(16, tmp_bytes), st));
    k_set_u32<<<1, 1, 0, st>>>(newdeg, n, 0);
    MG_CK(cub::DeviceScan::ExclusiveSum(tmp, tmp_bytes, newdeg, newoff, n + 1, st));
    cudaFreeAsync(tmp, st);
    k_compact_unique<<<grid_for(uint64_t(n) * 32, 256, dg->sms * 32), 256, 0, st>>>(off, sorted, n, newoff, adj);
    MG_CK(cudaMemcpyAsync(&mm, newoff + n, 4, cudaMemcpyDeviceToHost, st));
    cudaFreeAsync(sorted, st);
    cudaFreeAsync(newdeg, st);
    cudaFreeAsync(off, st);
    off = newoff;
    MG_CK(cudaStreamSynchronize(st));
  }
  uint32_t *adjL, *loff, *nlb, *deg;
  int rc;
  if ((rc = dev_alloc(dg, (void**)&adjL, uint64_t(std::max(mm, 1u)) * 4))) return rc;
  if ((rc = dev_alloc(dg, (void**)&loff, (uint64_t(n) * L + 1) * 4))) return rc;
  if ((rc = dev_alloc(dg, (void**)&nlb, uint64_t(n) * W * 4))) return rc;
  if ((rc = dev_alloc(dg, (void**)&deg, uint64_t(n) * 4))) return rc;
  const unsigned pt_grid = (n + PT_V - 1) / PT_V;
  const size_t hist_smem = size_t(L) * PT_STRIDE * 4;
  const size_t place_smem = hist_smem + size_t(PT_WARPS) * L * 4;
  const uint64_t slices = uint64_t(L) * n;
  const uint64_t tiles = (slices + SC_TILE - 1) / SC_TILE;
  uint32_t* sums = nullptr;
  MG_CK(cudaMallocAsync((void**)&sums, tiles * 4, st));
  k_label_count<<<pt_grid, PT_BLOCK, hist_smem, st>>>(off, adj, n, dg->g.input_id, d_label, L, W,
                                                      loff, nlb, deg,
                                                      const_cast<uint32_t*>(dg->g.selfbits));
  k_sum_tiles<<<unsigned(tiles), SC_BLOCK, 0, st>>>(loff, slices, sums);
  k_scan_sums<<<1, 1024, 0, st>>>(sums, uint32_t(tiles), loff + slices);
  k_scan_tiles<<<unsigned(tiles), SC_BLOCK, 0, st>>>(loff, slices, sums);
  k_label_scatter<<<pt_grid, PT_BLOCK, place_smem, st>>>(off, adj, n, dg->g.input_id, d_new,
                                                         d_label, L, loff, adjL);
  MG_CK(cudaGetLastError());
  cudaFreeAsync(sums, st);
  cudaFreeAsync(off, st);
  cudaFreeAsync(adj, st);
  dg->g.adj[d] = adjL;
  dg->g.loff[d] = loff;
  dg->g.nlb[d] = nlb;
  dg->g.deg[d] = deg;
  if (d == 0) dg->info.m_out = mm;
  else dg->info.m_in = mm;
  return MG_OK;
}

static int upload(const mg_csr_view* v, int device, const mg_upload_opts& uo, DevGraph* dg) {
  int rc = validate_csr_view(v);
  if (rc) return rc;
  if (v->n == 0) return set_error(MG_E_ARG, "empty data graph");
  int ndev = 0;
  MG_CK(cudaGetDeviceCount(&ndev));
  if (device < 0 || device >= ndev)
    return set_error(MG_E_ARG, "device %d not present (%d devices)", device, ndev);
  MG_CK(cudaSetDevice(device));
  dg->device = device;
  int sms = 0;
  MG_CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
  dg->sms = unsigned(std::max(sms, 1));
  MG_CK(cudaStreamCreateWithFlags(&dg->stream, cudaStreamNonBlocking));
  cudaStream_t st = dg->stream;
  const uint32_t n = v->n;
  dg->g.n = n;
  dg->info.n = n;
  dg->info.device = device;

  // Label compaction (host): distinct raw labels, ascending.  Small label
  // values (the usual case) are collected with a presence table in one pass;
  // other values by sorting a copy.
  std::vector<uint32_t> vals;
  {
    uint32_t lmax = 0;
    for (uint32_t i = 0; i < n; ++i) lmax = std::max(lmax, v->labels[i]);
    if (lmax < (1u << 22)) {
      std::vector<uint8_t> seen(uint64_t(lmax) + 1, 0);
      for (uint32_t i = 0; i < n; ++i) seen[v->labels[i]] = 1;
      for (uint32_t x = 0; x <= lmax; ++x)
        if (seen[x]) vals.push_back(x);
    } else {
      vals.assign(v->labels, v->labels + n);
      std::sort(vals.begin(), vals.end());
      vals.erase(std::unique(vals.begin(), vals.end()), vals.end());
    }
  }
  if (vals.size() > MG_MAX_LABELS)
    return set_error(MG_E_LIMIT, "%zu distinct labels; at most %d supported", vals.size(),
                     MG_MAX_LABELS);
  const uint32_t L = uint32_t(vals.size());
  const uint32_t W = (L + 31) / 32;
  dg->g.L = L;
  dg->g.W = W;
  dg->info.n_labels = L;
  dg->info.nlb_words = W;
  dg->stats.n = n;
  dg->stats.L = L;
  dg->stats.label_values = vals;
  std::vector<uint8_t> lab(n);  // compact labels, at most MG_MAX_LABELS
  std::vector<uint64_t> cnt(L, 0);
  if (vals.back() < (1u << 22)) {
    std::vector<uint32_t> to_compact(uint64_t(vals.back()) + 1, 0);
    for (uint32_t c = 0; c < L; ++c) to_compact[vals[c]] = c;
    for (uint32_t i = 0; i < n; ++i) {
      lab[i] = uint8_t(to_compact[v->labels[i]]);
      cnt[lab[i]]++;
    }
  } else {
    for (uint32_t i = 0; i < n; ++i) {
      lab[i] = uint8_t(std::lower_bound(vals.begin(), vals.end(), v->labels[i]) - vals.begin());
      cnt[lab[i]]++;
    }
  }
  dg->stats.label_count = cnt;
  dg->h_bucket_off.assign(L + 1, 0);
  for (uint32_t l = 0; l < L; ++l) dg->h_bucket_off[l + 1] = dg->h_bucket_off[l] + uint32_t(cnt[l]);
  // Vertices by (label, input id): input id of every vertex and the reverse.
  std::vector<uint32_t> input_id(n), new_id(n);
  {
    std::vector<uint32_t> cur(dg->h_bucket_off.begin(), dg->h_bucket_off.end() - 1);
    for (uint32_t i = 0; i < n; ++i) {
      new_id[i] = cur[lab[i]]++;
      input_id[new_id[i]] = i;
    }
  }
  uint8_t* d_label;
  uint32_t *d_boff, *d_input, *d_new, *d_self, *d_gid, *d_err;
  if ((rc = dev_alloc(dg, (void**)&d_boff, uint64_t(L + 1) * 4))) return rc;
  if ((rc = dev_alloc(dg, (void**)&d_input, uint64_t(n) * 4))) return rc;
  if ((rc = dev_alloc(dg, (void**)&d_self, uint64_t((n + 31) / 32) * 4))) return rc;
  if ((rc = dev_alloc(dg, (void**)&d_gid, uint64_t(n) * 4))) return rc;
  if ((rc = dev_alloc(dg, (void**)&d_err, 16))) return rc;
  MG_CK(cudaMallocAsync((void**)&d_label, uint64_t(n), st));
  MG_CK(cudaMallocAsync((void**)&d_new, uint64_t(n) * 4, st));
  MG_CK(cudaMemcpyAsync(d_label, lab.data(), uint64_t(n), cudaMemcpyHostToDevice, st));
  MG_CK(cudaMemcpyAsync(d_boff, dg->h_bucket_off.data(), uint64_t(L + 1) * 4,
                        cudaMemcpyHostToDevice, st));
  MG_CK(cudaMemcpyAsync(d_input, input_id.data(), uint64_t(n) * 4, cudaMemcpyHostToDevice, st));
  MG_CK(cudaMemcpyAsync(d_new, new_id.data(), uint64_t(n) * 4, cudaMemcpyHostToDevice, st));
  MG_CK(cudaMemsetAsync(d_self, 0, uint64_t((n + 31) / 32) * 4, st));
  MG_CK(cudaMemsetAsync(d_err, 0, 16, st));
  dg->g.bucket_off = d_boff;
  dg->g.input_id = d_input;
  dg->g.selfbits = d_self;
  dg->g.globalid = d_gid;

  // Global ids -> local ids when the stored ids are not the identity.
  bool ident = true;
  for (uint32_t i = 0; i < n && ident; ++i) ident = v->globalid[i] == i;
  dg->max_gid = ident ? n - 1 : v->max_vid;
  uint32_t* d_g2l = nullptr;
  if (ident) {
    MG_CK(cudaMemcpyAsync(d_gid, d_input, uint64_t(n) * 4, cudaMemcpyDeviceToDevice, st));
  } else {
    uint32_t* d_in_gid = nullptr;  // global ids in input order
    MG_CK(cudaMallocAsync((void**)&d_in_gid, uint64_t(n) * 4, st));
    MG_CK(cudaMemcpyAsync(d_in_gid, v->globalid, uint64_t(n) * 4, cudaMemcpyHostToDevice, st));
    MG_CK(cudaMallocAsync((void**)&d_g2l, (uint64_t(v->max_vid) + 1) * 4, st));
    MG_CK(cudaMemsetAsync(d_g2l, 0xFF, (uint64_t(v->max_vid) + 1) * 4, st));
    const unsigned grid = grid_for(n, 256, dg->sms * 32);
    k_build_g2l<<<grid, 256, 0, st>>>(d_in_gid, n, d_g2l, v->max_vid, d_err);
    k_permute_u32<<<grid, 256, 0, st>>>(d_in_gid, d_input, n, d_gid);
    cudaFreeAsync(d_in_gid, st);
  }
  const bool sym = v->m_in == v->m_out && arrays_equal(v->in_off, v->out_off, uint64_t(n) + 1) &&
                   arrays_equal(v->in_edges, v->out_edges, v->m_out);
  dg->g.symmetric = sym;
  dg->info.symmetric = sym;
  dg->stats.symmetric = sym;
  rc = build_direction(dg, 0, v->out_off, v->out_edges, v->m_out, d_g2l, v->max_vid, d_new, d_label,
                       d_err);
  if (rc == MG_OK) {
    if (sym) {
      dg->g.adj[1] = dg->g.adj[0];
      dg->g.loff[1] = dg->g.loff[0];
      dg->g.nlb[1] = dg->g.nlb[0];
      dg->g.deg[1] = dg->g.deg[0];
      dg->info.m_in = dg->info.m_out;
    } else {
      rc = build_direction(dg, 1, v->in_off, v->in_edges, v->m_in, d_g2l, v->max_vid, d_new, d_label,
                           d_err);
    }
  }
  if (d_g2l) cudaFreeAsync(d_g2l, st);
  cudaFreeAsync(d_label, st);
  cudaFreeAsync(d_new, st);
  if (rc) return rc;
  uint32_t err = 0;
  MG_CK(cudaMemcpyAsync(&err, d_err, 4, cudaMemcpyDeviceToHost, st));
  MG_CK(cudaStreamSynchronize(st));
  if (err & ERR_RANGE) return set_error(MG_E_FORMAT, "vertex id outside [0, max_vid] or unknown");
  // Maximum degree (host reduction over the reference outdeg is not trusted:
  // read the distinct-neighbour degrees back), then the hub bitmaps.
  uint64_t budget = uo.hub_bytes;
  if (budget == MG_HUB_AUTO) {
    size_t free_b = 0, total_b = 0;
    MG_CK(cudaMemGetInfo(&free_b, &total_b));
    budget = std::min<uint64_t>(4ull << 30, free_b / 8);
  }
  const uint32_t min_degree = uo.hub_min_degree ? uo.hub_min_degree : 128u;
  for (int d = 0; d < (sym ? 1 : 2); ++d) {
    std::vector<uint32_t> h(n);
    MG_CK(cudaMemcpy(h.data(), dg->g.deg[d], uint64_t(n) * 4, cudaMemcpyDeviceToHost));
    if (d == 0) dg->info.max_degree = *std::max_element(h.begin(), h.end());
    if (budget && (rc = build_hubs(dg, d, h, sym ? budget : budget / 2, min_degree))) return rc;
  }
  if (sym) {
    dg->g.hub_slot[1] = dg->g.hub_slot[0];
    dg->g.hub_bits[1] = dg->g.hub_bits[0];
  }
  return MG_OK;
}

int ensure_full_stats(DevGraph* dg) {
  if (dg->stats_full) return MG_OK;
  const uint32_t L = dg->g.L, n = dg->g.n;
  cudaStream_t st = dg->stream;
  unsigned long long *dsum, *dhist, *dpair;
  unsigned int* dmax;
  MG_CK(cudaMallocAsync((void**)&dsum, L * 8ull, st));
  MG_CK(cudaMallocAsync((void**)&dhist, L * 33 * 8ull, st));
  MG_CK(cudaMallocAsync((void**)&dpair, uint64_t(L) * L * 8, st));
  MG_CK(cudaMallocAsync((void**)&dmax, L * 4ull, st));
  MG_CK(cudaMemsetAsync(dsum, 0, L * 8ull, st));
  MG_CK(cudaMemsetAsync(dhist, 0, L * 33 * 8ull, st));
  MG_CK(cudaMemsetAsync(dpair, 0, uint64_t(L) * L * 8, st));
  MG_CK(cudaMemsetAsync(dmax, 0, L * 4ull, st));
  uint32_t widest = 1;  // largest label bucket
  for (uint32_t l = 0; l < L; ++l)
    widest = std::max(widest, dg->h_bucket_off[l + 1] - dg->h_bucket_off[l]);
  k_label_stats<<<dim3(grid_for(widest, LS_PART, 1024), L), 256, 0, st>>>(
      dg->g.loff[0], dg->g.deg[0], dg->g.bucket_off, n, L, dsum, dmax, dhist, dpair);
  std::vector<unsigned long long> hsum(L), hhist(L * 33), hpair(uint64_t(L) * L);
  std::vector<unsigned int> hmax(L);
  MG_CK(cudaMemcpyAsync(hsum.data(), dsum, L * 8ull, cudaMemcpyDeviceToHost, st));
  MG_CK(cudaMemcpyAsync(hhist.data(), dhist, L * 33 * 8ull, cudaMemcpyDeviceToHost, st));
  MG_CK(cudaMemcpyAsync(hpair.data(), dpair, uint64_t(L) * L * 8, cudaMemcpyDeviceToHost, st));
  MG_CK(cudaMemcpyAsync(hmax.data(), dmax, L * 4ull, cudaMemcpyDeviceToHost, st));
  MG_CK(cudaStreamSynchronize(st));
  cudaFreeAsync(dsum, st);
  cudaFreeAsync(dhist, st);
  cudaFreeAsync(dpair, st);
  cudaFreeAsync(dmax, st);
  auto& S = dg->stats;
  S.label_deg_mean.assign(L, 0);
  S.label_deg_max.assign(L, 0);
  S.label_deg_p99.assign(L, 0);
  S.label_pair_edges.assign(hpair.begin(), hpair.end());
  S.label_nlb_density.assign(L, 0);
  for (uint32_t l = 0; l < L; ++l) {
    uint64_t c = S.label_count[l];
    S.label_deg_mean[l] = c ? double(hsum[l]) / double(c) : 0.0;
    S.label_deg_max[l] = double(hmax[l]);
    uint64_t target = c - c / 100, acc = 0;
    for (uint32_t b = 0; b < 33; ++b) {
      acc += hhist[l * 33 + b];
      if (acc >= target && c) {
        S.label_deg_p99[l] = b == 0 ? 0.0 : double((1ull << b) - 1);
        break;
      }
    }
    uint64_t nl = 0;
    for (uint32_t l2 = 0; l2 < L; ++l2) nl += hpair[uint64_t(l) * L + l2] > 0;
    S.label_nlb_density[l] = nl;
  }
  dg->stats_full = true;
  return MG_OK;
}

// Device of an entry point that takes no device argument: the one named by
// MATRIXGRAPH_CUDA_DEVICE when it is a valid index (the reference's
// set_device_from_env, core/go_api/matrixgraph_go_api.cu:22-34), else the
// calling thread's current device.  The current device is not changed.
int env_or_current_device(int* dev) {
  int count = 0;
  MG_CK(cudaGetDeviceCount(&count));
  const char* s = std::getenv("MATRIXGRAPH_CUDA_DEVICE");
  if (s && s[0]) {
    const int d = std::atoi(s);
    if (d >= 0 && d < count) {
      *dev = d;
      return MG_OK;
    }
  }
  MG_CK(cudaGetDevice(dev));
  return MG_OK;
}

}  // namespace mg

extern "C" {

int mg_graph_upload(const mg_csr_view* g, int device, void** dgraph) {
  return mg_graph_upload_ex(g, device, nullptr, dgraph);
}

int mg_graph_upload_ex(const mg_csr_view* g, int device, const mg_upload_opts* opts,
                       void** dgraph) {
  mg::clear_error();
  if (!g || !dgraph) return mg::set_error(MG_E_ARG, "null argument");
  mg_upload_opts uo{MG_HUB_AUTO, 0, 0};
  if (opts) uo = *opts;
  if (uo._reserved) return mg::set_error(MG_E_ARG, "reserved upload option must be 0");
  auto* dg = new (std::nothrow) mg::DevGraph();
  if (!dg) return mg::set_error(MG_E_OOM, "host allocation failed");
  int prev = 0;
  cudaGetDevice(&prev);
  int rc;
  try {
    rc = mg::upload(g, device, uo, dg);
  } catch (const std::bad_alloc&) {
    rc = mg::set_error(MG_E_OOM, "host allocation failed");
  }
  cudaSetDevice(prev);
  if (rc) {
    delete dg;
    return rc;
  }
  *dgraph = dg;
  return MG_OK;
}

void mg_graph_free(void* dgraph) { delete static_cast<mg::DevGraph*>(dgraph); }

int mg_graph_get_info(void* dgraph, mg_graph_info* info) {
  mg::clear_error();
  if (!dgraph || !info) return mg::set_error(MG_E_ARG, "null argument");
  *info = static_cast<mg::DevGraph*>(dgraph)->info;
  return MG_OK;
}

}  // extern "C"
