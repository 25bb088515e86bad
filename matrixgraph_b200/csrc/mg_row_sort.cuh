// Lexicographic sort of emitted rows: rows are packed into 64-bit keys and
// sorted by a least-significant-digit radix sort of 8-bit digits.
//
// A row of k ids of b bits is one key when k * b <= 64; only the bits that ids
// can have are sorted, and the key is the whole row, so no index travels with
// it.  Wider rows are packed into several keys of as many columns as fit and
// sorted from the last one on, with a row index as payload.
//
//   k_sort_small   up to SS_MAX rows: every pass in one block and one launch
//   k_digit_hist / k_digit_scan / k_digit_pass
//                  more rows: the histograms of all digits in one pass over the
//                  keys, then one launch per digit (single-pass scatter with
//                  decoupled look-back per digit)
//
// The former sort took 32-bit columns with a row index through four passes
// each, five launches a pass.  Bound by launches for small results and by HBM
// (16 bytes read and written per key and pass) for large ones.
#pragma once

#include "mg_device.cuh"

namespace mg {

using u64 = unsigned long long;

constexpr int SS_BLOCK = 1024, SS_PER = 8, SS_MAX = SS_BLOCK * SS_PER;
constexpr int OS_BLOCK = 256, OS_PER = 8, OS_TILE = OS_BLOCK * OS_PER;
constexpr int DIGITS = 256, MAX_PASSES = 8;

__device__ __forceinline__ uint32_t lane_below() { return (1u << (threadIdx.x & 31)) - 1u; }

// Exclusive prefix sums of v over the first 256 threads (8 warps) of a block;
// the other threads pass through.  sums: 8 words of shared memory.
__device__ __forceinline__ uint32_t scan_digits(uint32_t v, uint32_t* sums) {
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t incl = v;
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t t = __shfl_up_sync(FULL, incl, d);
    if (lane >= uint32_t(d)) incl += t;
  }
  if (warp < 8 && lane == 31) sums[warp] = incl;
  __syncthreads();
  uint32_t before = 0;
  for (uint32_t w = 0; w < min(warp, 8u); ++w) before += sums[w];
  __syncthreads();
  return before + incl - v;
}

// Sorts n <= SS_MAX keys (and their payload) by their low `bits` bits, in place.
// Dynamic shared memory: SS_MAX keys, SS_MAX payloads when PAY, 32 x 256 counts.
template <bool PAY>
__global__ void __launch_bounds__(SS_BLOCK) k_sort_small(u64* keys, uint32_t* vals, uint32_t n,
                                                        uint32_t bits) {
  extern __shared__ __align__(16) unsigned char smem[];
  u64* sk = reinterpret_cast<u64*>(smem);
  uint32_t* sv = reinterpret_cast<uint32_t*>(sk + SS_MAX);
  uint16_t* cnt = reinterpret_cast<uint16_t*>(sv + (PAY ? SS_MAX : 0));
  __shared__ uint32_t base[DIGITS], sums[8];
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t per = (n + SS_BLOCK - 1) / SS_BLOCK;  // keys per thread
  const uint32_t first = warp * per * 32 + lane;
  u64 key[SS_PER];
  uint32_t val[SS_PER], rank[SS_PER];
#pragma unroll
  for (int r = 0; r < SS_PER; ++r) {
    const uint32_t i = first + r * 32;
    if (uint32_t(r) < per) {
      key[r] = i < n ? keys[i] : ~0ull;  // padding sorts last
      val[r] = PAY && i < n ? vals[i] : 0u;
    }
  }
  uint16_t* mine = cnt + warp * DIGITS;
  for (uint32_t shift = 0; shift < bits; shift += 8) {
    for (uint32_t d = lane; d < DIGITS; d += 32) mine[d] = 0;
    __syncwarp();
#pragma unroll
    for (int r = 0; r < SS_PER; ++r) {
      if (uint32_t(r) >= per) break;
      const uint32_t d = uint32_t(key[r] >> shift) & 255u;
      const uint32_t peers = __match_any_sync(FULL, d);
      const uint32_t below = __popc(peers & lane_below());
      const uint32_t at = mine[d];
      __syncwarp();
      if (below == 0) mine[d] = uint16_t(at + __popc(peers));
      __syncwarp();
      rank[r] = at + below;
    }
    __syncthreads();
    uint32_t total = 0;
    if (threadIdx.x < DIGITS)
      for (uint32_t w = 0; w < SS_BLOCK / 32; ++w) {
        const uint32_t c = cnt[w * DIGITS + threadIdx.x];
        cnt[w * DIGITS + threadIdx.x] = uint16_t(total);
        total += c;
      }
    const uint32_t ex = scan_digits(total, sums);
    if (threadIdx.x < DIGITS) base[threadIdx.x] = ex;
    __syncthreads();
#pragma unroll
    for (int r = 0; r < SS_PER; ++r) {
      if (uint32_t(r) >= per) break;
      const uint32_t d = uint32_t(key[r] >> shift) & 255u;
      const uint32_t at = base[d] + mine[d] + rank[r];
      sk[at] = key[r];
      if (PAY) sv[at] = val[r];
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < SS_PER; ++r) {
      if (uint32_t(r) >= per) break;
      key[r] = sk[first + r * 32];
      if (PAY) val[r] = sv[first + r * 32];
    }
  }
#pragma unroll
  for (int r = 0; r < SS_PER; ++r) {
    const uint32_t i = first + r * 32;
    if (uint32_t(r) < per && i < n) {
      keys[i] = key[r];
      if (PAY) vals[i] = val[r];
    }
  }
}

// Histograms of every digit: hist[pass * 256 + digit], zeroed before.
__global__ void __launch_bounds__(256) k_digit_hist(const u64* __restrict__ keys, uint64_t n,
                                                    uint32_t passes, u64* hist) {
  __shared__ uint32_t h[MAX_PASSES * DIGITS];
  for (uint32_t x = threadIdx.x; x < passes * DIGITS; x += blockDim.x) h[x] = 0;
  __syncthreads();
  for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < n;
       i += uint64_t(gridDim.x) * blockDim.x) {
    const u64 k = keys[i];
    for (uint32_t p = 0; p < passes; ++p)
      atomicAdd(&h[p * DIGITS + (uint32_t(k >> (8 * p)) & 255u)], 1u);
  }
  __syncthreads();
  for (uint32_t x = threadIdx.x; x < passes * DIGITS; x += blockDim.x)
    if (h[x]) atomicAdd(&hist[x], u64(h[x]));
}

// Exclusive prefix sums of each pass's histogram (one block, a pass per warp).
__global__ void __launch_bounds__(MAX_PASSES * 32) k_digit_scan(u64* hist, uint32_t passes) {
  const uint32_t lane = threadIdx.x & 31, p = threadIdx.x >> 5;
  if (p >= passes) return;
  u64 carry = 0;
  for (uint32_t d0 = 0; d0 < DIGITS; d0 += 32) {
    const u64 v = hist[p * DIGITS + d0 + lane];
    u64 incl = v;
    for (int d = 1; d < 32; d <<= 1) {
      const u64 t = __shfl_up_sync(FULL, incl, d);
      if (lane >= uint32_t(d)) incl += t;
    }
    hist[p * DIGITS + d0 + lane] = carry + incl - v;
    carry += __shfl_sync(FULL, incl, 31);
  }
}

// One stable pass over digit `pass`: tiles are claimed in order, each ranks its
// keys, publishes its digit counts, adds the counts of the tiles before it
// (one digit per thread; words [epoch:8 | state:2 | count:54]) and writes its
// keys, grouped by digit, to their places.  A tile waits only for tiles claimed
// before it, at most spin_limit polls (ERR_TIMEOUT in *err).
constexpr u64 DS_SUM = 1, DS_PREFIX = 2;
__device__ __forceinline__ u64 ds_word(uint32_t epoch, u64 state, u64 v) {
  return u64(epoch) << 56 | state << 54 | v;
}

template <bool PAY>
__global__ void __launch_bounds__(OS_BLOCK) k_digit_pass(
    const u64* __restrict__ keys, const uint32_t* __restrict__ vals, u64* keys_out,
    uint32_t* vals_out, uint64_t n, uint32_t pass, const u64* __restrict__ base, u64* status,
    u64* claim, uint32_t spin_limit, u64* err) {
  __shared__ u64 sk[OS_TILE];
  __shared__ uint32_t sv[PAY ? OS_TILE : 1];
  __shared__ uint32_t cnt[OS_BLOCK / 32][DIGITS];
  __shared__ uint32_t lofs[DIGITS], sums[8];
  __shared__ u64 gofs[DIGITS];
  __shared__ uint32_t s_tile;
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, me = threadIdx.x;
  const uint32_t epoch = pass + 1, shift = pass * 8;
  if (me == 0) s_tile = uint32_t(atomicAdd(claim, 1ull));
  for (uint32_t d = lane; d < DIGITS; d += 32) cnt[warp][d] = 0;
  __syncthreads();
  const uint64_t tile = s_tile, first = tile * OS_TILE + warp * (32 * OS_PER) + lane;
  u64 key[OS_PER];
  uint32_t val[OS_PER], rank[OS_PER];
#pragma unroll
  for (int r = 0; r < OS_PER; ++r) {
    const uint64_t i = first + r * 32;
    key[r] = i < n ? keys[i] : 0ull;
    val[r] = PAY && i < n ? vals[i] : 0u;
  }
#pragma unroll
  for (int r = 0; r < OS_PER; ++r) {
    const bool valid = first + r * 32 < n;
    const uint32_t d = uint32_t(key[r] >> shift) & 255u;
    const uint32_t peers = __match_any_sync(FULL, valid ? d : DIGITS + lane);
    const uint32_t below = __popc(peers & lane_below());
    const uint32_t at = valid ? cnt[warp][d] : 0u;
    __syncwarp();
    if (valid && below == 0) cnt[warp][d] = at + __popc(peers);
    __syncwarp();
    rank[r] = at + below;
  }
  __syncthreads();
  uint32_t total = 0;
  for (uint32_t w = 0; w < OS_BLOCK / 32; ++w) {
    const uint32_t c = cnt[w][me];
    cnt[w][me] = total;
    total += c;
  }
  volatile u64* st = status;
  st[tile * DIGITS + me] = ds_word(epoch, tile ? DS_SUM : DS_PREFIX, total);
  const uint32_t lo = scan_digits(total, sums);
  lofs[me] = lo;
  u64 prefix = 0;
  for (int64_t t = int64_t(tile) - 1; t >= 0; --t) {
    u64 w = 0;
    uint32_t spins = 0;
    for (;;) {
      w = st[t * DIGITS + me];
      if (w >> 56 == epoch) break;
      if (++spins > spin_limit) {
        atomicOr(err, u64(ERR_TIMEOUT));
        w = ds_word(epoch, DS_PREFIX, 0);
        break;
      }
      __nanosleep(32);
    }
    prefix += w & ((1ull << 54) - 1);
    if ((w >> 54 & 3ull) == DS_PREFIX) break;
  }
  if (tile) st[tile * DIGITS + me] = ds_word(epoch, DS_PREFIX, prefix + total);
  gofs[me] = base[pass * DIGITS + me] + prefix - lo;
  __syncthreads();
#pragma unroll
  for (int r = 0; r < OS_PER; ++r) {
    if (first + r * 32 >= n) continue;
    const uint32_t d = uint32_t(key[r] >> shift) & 255u;
    const uint32_t at = lofs[d] + cnt[warp][d] + rank[r];
    sk[at] = key[r];
    if (PAY) sv[at] = val[r];
  }
  __syncthreads();
  const uint32_t held = uint32_t(min(uint64_t(OS_TILE), n - tile * OS_TILE));
  for (uint32_t x = me; x < held; x += OS_BLOCK) {
    const u64 k = sk[x];
    const u64 at = gofs[uint32_t(k >> shift) & 255u] + x;
    if (at >= n) continue;  // only after a wait that gave up
    keys_out[at] = k;
    if (PAY) vals_out[at] = sv[x];
  }
}

__global__ void k_iota(uint32_t* p, uint64_t n) {
  for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < n;
       i += uint64_t(gridDim.x) * blockDim.x)
    p[i] = uint32_t(i);
}

// Columns [c0, c1) of every row in the order of perm, packed with b bits each.
struct RowCols {
  const uint32_t* col[MAXK];
};
__global__ void k_pack_cols(RowCols cols, uint32_t c0, uint32_t c1, uint32_t b,
                            const uint32_t* __restrict__ perm, uint64_t n, u64* keys) {
  for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < n;
       i += uint64_t(gridDim.x) * blockDim.x) {
    const uint32_t r = perm[i];
    u64 k = 0;
    for (uint32_t c = c0; c < c1; ++c) k = k << b | cols.col[c][r];
    keys[i] = k;
  }
}

// Row-major output of the first n rows: from packed keys, or from the columns.
__global__ void k_rows_from_keys(const u64* __restrict__ keys, uint32_t k, uint32_t b, uint64_t n,
                                 uint32_t* rows) {
  const u64 mask = b == 64 ? ~0ull : (1ull << b) - 1;
  for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < n * k;
       i += uint64_t(gridDim.x) * blockDim.x) {
    const uint64_t r = i / k;
    const uint32_t c = uint32_t(i - r * k);
    rows[i] = uint32_t(keys[r] >> ((k - 1 - c) * b) & mask);
  }
}

__global__ void k_rows_from_cols(RowCols cols, const uint32_t* __restrict__ perm, uint32_t k,
                                 uint64_t n, uint32_t* rows) {
  for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < n * k;
       i += uint64_t(gridDim.x) * blockDim.x) {
    const uint64_t r = i / k;
    rows[i] = cols.col[i - r * k][perm[r]];
  }
}

// Memory of an emit call, carved out of one block: room for `cap` rows.
struct RowBuf {
  uint32_t k = 0, bits = 0;  // ids per row, bits per id
  uint64_t cap = 0;
  bool packed = false;  // a row is one key
  u64 *key_a = nullptr, *key_b = nullptr;
  uint32_t *val_a = nullptr, *val_b = nullptr;
  uint32_t* col[MAXK] = {};
  uint32_t* rows = nullptr;
  u64* hist = nullptr;    // MAX_PASSES * 256, then MAX_PASSES claims, then the error word
  u64* status = nullptr;  // 256 words per tile
  static constexpr uint64_t kHead = MAX_PASSES * DIGITS + MAX_PASSES + 1;

  // Lays the arrays out from `base` (nullptr: only measures) and returns their
  // bytes.
  uint64_t carve(unsigned char* base, uint32_t k_, uint32_t bits_, uint64_t cap_) {
    k = k_;
    bits = bits_;
    cap = cap_;
    packed = k * bits <= 64;
    uint64_t off = 0;
    auto take = [&](uint64_t bytes) {
      off = (off + 255) & ~uint64_t(255);
      unsigned char* p = base ? base + off : nullptr;
      off += bytes;
      return p;
    };
    const uint64_t rows_ = cap ? cap : 1;
    hist = reinterpret_cast<u64*>(take(kHead * 8));
    status = reinterpret_cast<u64*>(take((rows_ + OS_TILE - 1) / OS_TILE * DIGITS * 8));
    key_a = reinterpret_cast<u64*>(take(rows_ * 8));
    key_b = reinterpret_cast<u64*>(take(rows_ * 8));
    rows = reinterpret_cast<uint32_t*>(take(rows_ * k * 4));
    if (!packed) {
      val_a = reinterpret_cast<uint32_t*>(take(rows_ * 4));
      val_b = reinterpret_cast<uint32_t*>(take(rows_ * 4));
      for (uint32_t c = 0; c < k; ++c) col[c] = reinterpret_cast<uint32_t*>(take(rows_ * 4));
    }
    return off;
  }
};

// Sorts the n keys of key_a by their low `bits` bits, with val_a as payload when
// PAY (results in key_a / val_a again).
template <bool PAY>
inline int sort_keys(RowBuf& B, uint64_t n, uint32_t bits, unsigned sms, uint32_t spin_limit,
                     cudaStream_t st) {
  if (n < 2 || bits == 0) return MG_OK;
  if (n <= SS_MAX) {
    const size_t smem = SS_MAX * (8 + (PAY ? 4 : 0)) + (SS_BLOCK / 32) * DIGITS * 2;
    MG_CK(cudaFuncSetAttribute(k_sort_small<PAY>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               int(smem)));
    k_sort_small<PAY><<<1, SS_BLOCK, smem, st>>>(B.key_a, B.val_a, uint32_t(n), bits);
    MG_CK(cudaGetLastError());
    return MG_OK;
  }
  const uint32_t passes = (bits + 7) / 8;
  const uint64_t tiles = (n + OS_TILE - 1) / OS_TILE;
  u64* claims = B.hist + MAX_PASSES * DIGITS;
  MG_CK(cudaMemsetAsync(B.hist, 0, (RowBuf::kHead - 1) * 8, st));
  MG_CK(cudaMemsetAsync(B.status, 0, tiles * DIGITS * 8, st));
  k_digit_hist<<<unsigned(std::min<uint64_t>(sms * 4, (n + 1023) / 1024)), 256, 0, st>>>(
      B.key_a, n, passes, B.hist);
  k_digit_scan<<<1, MAX_PASSES * 32, 0, st>>>(B.hist, passes);
  for (uint32_t p = 0; p < passes; ++p) {
    k_digit_pass<PAY><<<unsigned(tiles), OS_BLOCK, 0, st>>>(
        B.key_a, B.val_a, B.key_b, B.val_b, n, p, B.hist, B.status, claims + p, spin_limit,
        claims + MAX_PASSES);
    std::swap(B.key_a, B.key_b);
    std::swap(B.val_a, B.val_b);
  }
  MG_CK(cudaGetLastError());
  return MG_OK;
}

// Sorts the n emitted rows of B and copies the first n_copy of them to h_rows
// (row-major, host).
inline int sort_rows(RowBuf& B, uint64_t n, uint64_t n_copy, uint32_t* h_rows, unsigned sms,
                     uint32_t spin_limit, cudaStream_t st) {
  if (n == 0 || n_copy == 0) return MG_OK;
  auto grid = [&](uint64_t items) {
    return unsigned(std::max<uint64_t>(1, std::min<uint64_t>((items + 255) / 256, 4096)));
  };
  u64* err = B.hist + RowBuf::kHead - 1;
  MG_CK(cudaMemsetAsync(err, 0, 8, st));
  int rc;
  if (B.packed) {
    if ((rc = sort_keys<false>(B, n, B.k * B.bits, sms, spin_limit, st))) return rc;
    k_rows_from_keys<<<grid(n_copy * B.k), 256, 0, st>>>(B.key_a, B.k, B.bits, n_copy, B.rows);
  } else {
    RowCols cols{};
    for (uint32_t c = 0; c < B.k; ++c) cols.col[c] = B.col[c];
    k_iota<<<grid(n), 256, 0, st>>>(B.val_a, n);
    const uint32_t per = 64 / B.bits;
    for (uint32_t c1 = B.k; c1 > 0;) {
      const uint32_t c0 = c1 > per ? c1 - per : 0;
      k_pack_cols<<<grid(n), 256, 0, st>>>(cols, c0, c1, B.bits, B.val_a, n, B.key_a);
      if ((rc = sort_keys<true>(B, n, (c1 - c0) * B.bits, sms, spin_limit, st))) return rc;
      c1 = c0;
    }
    k_rows_from_cols<<<grid(n_copy * B.k), 256, 0, st>>>(cols, B.val_a, B.k, n_copy, B.rows);
  }
  MG_CK(cudaGetLastError());
  u64 e = 0;
  MG_CK(cudaMemcpyAsync(&e, err, 8, cudaMemcpyDeviceToHost, st));
  MG_CK(cudaMemcpyAsync(h_rows, B.rows, n_copy * B.k * 4, cudaMemcpyDeviceToHost, st));
  MG_CK(cudaStreamSynchronize(st));
  if (e & ERR_TIMEOUT) return set_error(MG_E_TIMEOUT, "row sort: a device wait gave up");
  return MG_OK;
}

}  // namespace mg
