// partition.cuh — stable counting-sort passes over (key, index, value) entries.
//
// One pass sorts by up to 10 bits of an int32 key: per-tile digit counts, a
// scan per digit over the tiles, and a scatter in which a CTA ranks its tile
// by digit in shared memory and writes every digit's run in one piece.  A
// matrix of 2^20 columns takes two passes, least significant digit first, so
// every entry crosses memory four times and nothing is sorted per segment.
//
// What bounds it: the scatter (reads 16 bytes an entry and writes 16 in runs
// of ~8 entries; ranks by a ballot per digit bit, which is several times the
// rate of __match_any_sync).
#pragma once

#include <algorithm>

#include "internal.cuh"

namespace tspg {

constexpr int kPartThreads = 512;
constexpr int kPartWarps = kPartThreads / 32;
constexpr int kPartBits = 10;  // digit width: 1024 counters per warp

// The entries a pass works on: `count` of them, or, when they are a CSR's
// (rp given), those its offsets span (a view's offsets need not start at 0 and
// its count may be an upper bound).
struct PartSpan {
  int64_t count = 0;
  const void *rp = nullptr;
  int32_t rp_bits = 64;
  int64_t m = 0;
  __device__ __forceinline__ int64_t at(int64_t i) const {
    return rp_bits == 32 ? int64_t(((const int32_t *)rp)[i]) : ((const int64_t *)rp)[i];
  }
  __device__ __forceinline__ int64_t base() const { return rp ? at(0) : 0; }
  __device__ __forceinline__ int64_t live() const {
    if (!rp) return count;
    const int64_t n = at(m) - at(0);
    return n < count ? n : count;
  }
};

// Digit counts of every tile: table[tile << bits | digit].
template <int ITEMS>
__global__ void __launch_bounds__(kPartThreads)
    k_part_count(const int32_t *key, PartSpan S, bool source, int shift, int bits, uint32_t *table) {
  __shared__ uint32_t cnt[1 << kPartBits];
  const int tid = threadIdx.x, nd = 1 << bits;
  const int64_t count = S.live();
  if (source) key += S.base();
  for (int d = tid; d < nd; d += kPartThreads) cnt[d] = 0;
  __syncthreads();
  const int64_t e0 = int64_t(blockIdx.x) * kPartThreads * ITEMS;
#pragma unroll
  for (int it = 0; it < ITEMS; ++it) {
    const int64_t e = e0 + it * kPartThreads + tid;
    if (e < count) atomicAdd(cnt + ((uint32_t(key[e]) >> shift) & (nd - 1)), 1u);
  }
  __syncthreads();
  for (int d = tid; d < nd; d += kPartThreads) table[(int64_t(blockIdx.x) << bits) + d] = cnt[d];
}

// Exclusive scan over the tiles of every digit's counts, in place; the digits'
// totals go to dtotal.  A CTA takes 8 digits (one sector of the table per
// tile): its threads are 128 streams of consecutive tiles x
// 8 digits.  (32 digits a CTA left it at 32 CTAs: 28 us for 3300 tiles.)
constexpr int kPartScanThreads = 1024;
static __global__ void __launch_bounds__(kPartScanThreads)
    k_part_scan(uint32_t *table, int64_t ntiles, int bits, uint32_t *dtotal) {
  constexpr int NS = kPartScanThreads / 8, U = 8;
  __shared__ uint32_t sum[8][NS + 1];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int dl = threadIdx.x & 7, st = threadIdx.x >> 3, d = blockIdx.x * 8 + dl;
  const bool have = d < (1 << bits);
  const int64_t per = (ntiles + NS - 1) / NS, t0 = st * per;
  const int64_t t1 = t0 + per < ntiles ? t0 + per : ntiles;
  uint32_t *col = table + d;
  uint32_t s = 0;
  for (int64_t t = t0; t < t1; t += U) {
    uint32_t v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) v[u] = have && t + u < t1 ? col[(t + u) << bits] : 0u;
#pragma unroll
    for (int u = 0; u < U; ++u) s += v[u];
  }
  sum[dl][st] = s;
  __syncthreads();
  if (w < 8) {  // warp w: digit w's 128 sums, 4 per lane
    uint32_t x[4], mine = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      x[k] = sum[w][lane * 4 + k];
      mine += x[k];
    }
    const uint32_t inc = warp_scan_incl(mine);
    uint32_t run = inc - mine;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      sum[w][lane * 4 + k] = run;
      run += x[k];
    }
    if (lane == 31 && blockIdx.x * 8 + w < (1 << bits)) dtotal[blockIdx.x * 8 + w] = inc;
  }
  __syncthreads();
  uint32_t run = sum[dl][st];
  for (int64_t t = t0; t < t1; t += U) {
    uint32_t v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) v[u] = have && t + u < t1 ? col[(t + u) << bits] : 0u;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (have && t + u < t1) col[(t + u) << bits] = run;
      run += v[u];
    }
  }
}

// Dynamic shared memory of k_part_scatter: the tile's keys in digit order, a
// staging buffer for one value array (the warps' digit counters before that)
// and the digits' output bases.
template <int ITEMS, typename VT>
__host__ __device__ constexpr uint32_t part_smem() {
  constexpr uint32_t T = kPartThreads * ITEMS;
  constexpr uint32_t buf = T * uint32_t(sizeof(VT)), cnt = kPartWarps * (1u << kPartBits) * 2u;
  return T * 4u + (buf > cnt ? buf : cnt) + (1u << kPartBits) * 4u;
}

// Scatter of a tile (source: key and val are the CSR's own arrays, idx the
// expanded rows).  Warp w owns entries [w * 32 ITEMS, (w + 1) * 32 ITEMS)
// of the tile in order, so ranks by (warp, item, lane) are stable.
template <int ITEMS, typename VT>
__global__ void __launch_bounds__(kPartThreads, 2)
    k_part_scatter(const int32_t *__restrict__ key, const int32_t *__restrict__ idx,
                   const VT *__restrict__ val, PartSpan S, bool source, int shift, int bits,
                   const uint32_t *__restrict__ table, const uint32_t *__restrict__ dtotal,
                   int32_t *__restrict__ okey, int32_t *__restrict__ oidx,
                   VT *__restrict__ oval) {
  constexpr int T = kPartThreads * ITEMS, ND = 1 << kPartBits;
  constexpr unsigned FULL = 0xffffffffu;
  extern __shared__ __align__(16) unsigned char sm[];
  int32_t *sk = (int32_t *)sm;
  unsigned char *buf = sm + T * 4;
  uint32_t *cnt = (uint32_t *)buf;  // [warp][digit pair], uint16 each
  uint16_t *c16 = (uint16_t *)buf;
  uint32_t *gb = (uint32_t *)(sm + part_smem<ITEMS, VT>() - ND * 4);
  __shared__ uint32_t tmp[2 * kPartWarps + 2];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const uint32_t dmask = (1u << bits) - 1u;
  const int64_t e0 = int64_t(blockIdx.x) * T;
  const int64_t left = S.live() - e0;  // may be negative past a view's end
  const int n = int(left < 0 ? 0 : left < T ? left : T);
  const int my = w * 32 * ITEMS + lane;
  const int64_t base = source ? S.base() : 0;
  key += base + e0 + my;
  idx += e0 + my;
  val += base + e0 + my;
  int32_t k[ITEMS];
#pragma unroll
  for (int it = 0; it < ITEMS; ++it) k[it] = my + it * 32 < n ? key[it * 32] : 0;
  for (int i = tid; i < kPartWarps * ND / 8; i += kPartThreads)
    ((uint4 *)buf)[i] = make_uint4(0, 0, 0, 0);
  __syncthreads();
  // rank within (warp, digit); lanes past the tile's end match nobody
  uint16_t pos[ITEMS];
  const unsigned lt = (1u << lane) - 1u;
#pragma unroll
  for (int it = 0; it < ITEMS; ++it) {
    const bool in = my + it * 32 < n;
    const uint32_t d = (uint32_t(k[it]) >> shift) & dmask;
    unsigned m = __ballot_sync(FULL, in);
#pragma unroll
    for (int b = 0; b < kPartBits; ++b) {  // bits past the digit's are 0 in every lane
      const bool one = d & (1u << b);
      const unsigned v = __ballot_sync(FULL, one);
      m &= one ? v : ~v;
    }
    uint16_t *c = c16 + w * ND + d;
    const int old = in ? *c : 0;
    __syncwarp();
    if (in && (m & lt) == 0) *c = uint16_t(old + __popc(m));
    __syncwarp();
    pos[it] = uint16_t(old + __popc(m & lt));
  }
  __syncthreads();
  // thread t: digits 2t and 2t + 1 over the warps, then over the digits
  uint32_t run = 0;  // packed pair
#pragma unroll
  for (int i = 0; i < kPartWarps; ++i) {
    const uint32_t v = cnt[i * (ND / 2) + tid];
    cnt[i * (ND / 2) + tid] = run;
    run += v;
  }
  const uint32_t lo = run & 0xffffu, hi = run >> 16;
  const uint32_t g0 = 2 * tid < int(dmask) + 1 ? dtotal[2 * tid] : 0u;
  const uint32_t g1 = 2 * tid + 1 < int(dmask) + 1 ? dtotal[2 * tid + 1] : 0u;
  const uint32_t sl = warp_scan_incl(lo + hi), sg = warp_scan_incl(g0 + g1);
  if (lane == 31) {
    tmp[w] = sl;
    tmp[kPartWarps + w] = sg;
  }
  __syncthreads();
  uint32_t bl = sl - lo - hi, bg = sg - g0 - g1;
  for (int i = 0; i < w; ++i) {
    bl += tmp[i];
    bg += tmp[kPartWarps + i];
  }
  // local digit bases into the counters, global ones (less the local) into gb
  const uint32_t pair = bl | ((bl + lo) << 16);
#pragma unroll
  for (int i = 0; i < kPartWarps; ++i) cnt[i * (ND / 2) + tid] += pair;
  if (2 * tid <= int(dmask)) {
    const uint2 before =
        *(const uint2 *)(table + (int64_t(blockIdx.x) << bits) + 2 * tid);  // bits >= 1
    gb[2 * tid] = bg + before.x - bl;
    gb[2 * tid + 1] = bg + g0 + before.y - (bl + lo);
  }
  __syncthreads();
#pragma unroll
  for (int it = 0; it < ITEMS; ++it) {
    if (my + it * 32 < n) {
      pos[it] = uint16_t(pos[it] + c16[w * ND + ((uint32_t(k[it]) >> shift) & dmask)]);
      sk[pos[it]] = k[it];
    }
  }
  __syncthreads();  // the counters' space is the staging buffer from here on
  auto slot = [&](int i) { return gb[(uint32_t(sk[i]) >> shift) & dmask] + uint32_t(i); };
  int32_t *si = (int32_t *)buf;
#pragma unroll
  for (int it = 0; it < ITEMS; ++it)
    if (my + it * 32 < n) si[pos[it]] = idx[it * 32];
  __syncthreads();
  for (int i = tid; i < n; i += kPartThreads) {
    const uint32_t o = slot(i);
    okey[o] = sk[i];
    oidx[o] = si[i];
  }
  __syncthreads();
  VT *sv = (VT *)buf;
#pragma unroll
  for (int it = 0; it < ITEMS; ++it)
    if (my + it * 32 < n) sv[pos[it]] = val[it * 32];
  __syncthreads();
  for (int i = tid; i < n; i += kPartThreads) oval[slot(i)] = sv[i];
}

// Row of every entry of a CSR (entries [0, count), positions rp[0] + e), a
// warp per kExpandRun entries.
constexpr int kExpandRun = 256;
template <typename PT>
__global__ void __launch_bounds__(256)
    k_expand_rows(const PT *__restrict__ rp, PartSpan S, int32_t *__restrict__ row) {
  const int64_t m = S.m, count = S.live();
  const int lane = threadIdx.x & 31;
  const int64_t w0 = ((int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5) * kExpandRun;
  if (w0 >= count) return;
  const int64_t base = int64_t(rp[0]);
  const int64_t w1 = w0 + kExpandRun < count ? w0 + kExpandRun : count;
  int64_t r = first_row(rp, m, base, w0, lane);
  for (int64_t e0 = w0; e0 < w1; e0 += 32) {
    const int64_t e = e0 + lane;
    const int64_t mine = window_row(rp, m, base, r, e, lane);
    if (e < w1) row[e] = int32_t(mine);
  }
}

// Offsets of the segments of sorted keys: ptr[k] = entries with a key below k.
// Entry e writes the offsets of the keys after its predecessor's up to its own
// (long gaps by the whole warp), entry `count` those past the last.  A warp
// takes 256 consecutive entries, all its loads in flight.
template <typename OT>
__global__ void __launch_bounds__(256)
    k_key_offsets(const int32_t *__restrict__ key, PartSpan S, int64_t n, OT *__restrict__ ptr) {
  const int64_t count = S.live();
  constexpr unsigned FULL = 0xffffffffu;
  constexpr int U = 8;
  const int lane = threadIdx.x & 31;
  const int64_t w0 = ((int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5) * (32 * U);
  if (w0 > count) return;
  int32_t k[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const int64_t e = w0 + u * 32 + lane;
    k[u] = e < count ? __ldg(key + e) : 0;
  }
  const int32_t before = w0 > 0 ? __ldg(key + w0 - 1) : -1;
  int32_t last = before;  // key of the entry before lane 0's
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const int64_t e = w0 + u * 32 + lane;
    const int32_t up = __shfl_up_sync(FULL, k[u], 1);
    int64_t a = int64_t(lane > 0 ? up : last) + 1, b = 0;  // ptr[a, b) = e
    last = __shfl_sync(FULL, k[u], 31);
    if (e < count) b = int64_t(k[u]) + 1;
    else if (e == count) b = n + 1;
    if (a < 0) a = 0;  // keys outside [0, n) write nothing out of range
    if (b > n + 1) b = n + 1;
    const bool wide = b - a > 8;
    if (!wide)
      for (int64_t q = a; q < b; ++q) ptr[q] = OT(e);
    for (unsigned todo = __ballot_sync(FULL, wide); todo; todo &= todo - 1) {
      const int j = __ffs(todo) - 1;
      const int64_t aj = __shfl_sync(FULL, a, j), bj = __shfl_sync(FULL, b, j);
      for (int64_t q = aj + lane; q < bj; q += 32) ptr[q] = OT(w0 + u * 32 + j);
    }
  }
}

// The same by a search per offset, for far more segments than entries.
template <typename OT>
__global__ void __launch_bounds__(256)
    k_key_offsets_sparse(const int32_t *__restrict__ key, PartSpan S, int64_t n,
                         OT *__restrict__ ptr) {
  const int64_t count = S.live();
  for (int64_t k = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; k <= n;
       k += int64_t(gridDim.x) * blockDim.x) {
    int64_t lo = 0, hi = count;
    while (lo < hi) {
      const int64_t mid = (lo + hi) >> 1;
      if (key[mid] < k) lo = mid + 1; else hi = mid;
    }
    ptr[k] = OT(lo);
  }
}

// ---------------------------------------------------------------- host side

constexpr int64_t kPartMaxEntries = INT64_C(0xffffffff);  // 32-bit positions
constexpr int64_t kPartBigTiles = 148 * 2 * 4;            // 8192-entry tiles worth having

inline int key_bits(int64_t n) {
  int b = 1;
  while (b < 32 && (int64_t(1) << b) < n) ++b;
  return b;
}
inline int part_passes(int64_t n) { return (key_bits(n) + kPartBits - 1) / kPartBits; }

struct PartScratch {
  uint32_t *table = nullptr, *dtotal = nullptr;
  int64_t ntiles = 0, table_len = 0;
  bool big = false;
};

inline void part_sizes(int64_t count, PartScratch *P) {
  const int64_t T16 = kPartThreads * 16, T4 = kPartThreads * 4;
  P->big = count >= kPartBigTiles * T16 / 4;
  const int64_t T = P->big ? T16 : T4;
  P->ntiles = (count + T - 1) / T;
  P->table_len = P->ntiles << kPartBits;
}

template <int ITEMS, typename VT>
inline int part_pass_t(tspg_ctx *ctx, cudaStream_t s, const PartScratch &P, const PartSpan &S,
                       bool source, int shift, int bits, const int32_t *key, const int32_t *idx, const VT *val,
                       int32_t *okey, int32_t *oidx, VT *oval) {
  constexpr uint32_t bytes = part_smem<ITEMS, VT>();
  const uint32_t mine = 16u << ((ITEMS == 16 ? 2 : 0) + (sizeof(VT) == 8 ? 1 : 0));
  if (!(ctx->smem_raised & mine)) {
    TSPG_CUDA(ctx, cudaFuncSetAttribute(k_part_scatter<ITEMS, VT>,
                                        cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
    ctx->smem_raised |= mine;
  }
  const unsigned g = unsigned(P.ntiles);
  k_part_count<ITEMS><<<g, kPartThreads, 0, s>>>(key, S, source, shift, bits, P.table);
  k_part_scan<<<((1u << bits) + 7) / 8, kPartScanThreads, 0, s>>>(P.table, P.ntiles, bits, P.dtotal);
  k_part_scatter<ITEMS, VT><<<g, kPartThreads, bytes, s>>>(key, idx, val, S, source, shift, bits, P.table,
                                                          P.dtotal, okey, oidx, oval);
  ctx->launches += 3;
  TSPG_CUDA(ctx, cudaGetLastError());
  return TSPG_OK;
}

// One stable pass by bits [shift, shift + bits) of key.  Tiles of 8192 entries
// (runs of ~8 per digit) when they fill the chip, else of 2048.
template <typename VT>
inline int part_pass(tspg_ctx *ctx, cudaStream_t s, const PartScratch &P, const PartSpan &S,
                     bool source, int shift, int bits, const int32_t *key, const int32_t *idx, const VT *val, int32_t *okey,
                     int32_t *oidx, VT *oval) {
  return P.big ? part_pass_t<16, VT>(ctx, s, P, S, source, shift, bits, key, idx, val, okey, oidx, oval)
               : part_pass_t<4, VT>(ctx, s, P, S, source, shift, bits, key, idx, val, okey, oidx, oval);
}

// Offsets (n + 1, `obits` wide) of the segments of sorted keys in [0, n).
inline int key_offsets(tspg_ctx *ctx, cudaStream_t s, const int32_t *key, const PartSpan &S, int64_t n,
                       void *ptr, int obits) {
  const int64_t count = S.count;
  const bool sparse = n > 8 * count;
  const unsigned g = sparse ? unsigned(std::min<int64_t>((n + 256) / 256, int64_t(ctx->num_sms) * 32))
                            : unsigned((count + 2048) / 2048);
  if (sparse) {
    if (obits == 32) k_key_offsets_sparse<int32_t><<<g, 256, 0, s>>>(key, S, n, (int32_t *)ptr);
    else k_key_offsets_sparse<int64_t><<<g, 256, 0, s>>>(key, S, n, (int64_t *)ptr);
  } else {
    if (obits == 32) k_key_offsets<int32_t><<<g, 256, 0, s>>>(key, S, n, (int32_t *)ptr);
    else k_key_offsets<int64_t><<<g, 256, 0, s>>>(key, S, n, (int64_t *)ptr);
  }
  ctx->launches += 1;
  TSPG_CUDA(ctx, cudaGetLastError());
  return TSPG_OK;
}

}  // namespace tspg
