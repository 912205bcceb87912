// spgemm_span.cuh — rows worked by one CTA with the whole column span in a
// shared-memory bitmap and the row's output in shared memory.
//
// A row takes five steps: its products mark their columns in the bitmap (a
// product that sets a new bit also counts it in its 128-column unit), a scan
// of the unit counters gives every unit its rank base, each product finds its
// output slot as base + popc of the bits below it and is added there in
// shared memory (the column is stored with it), and the slots leave for C in
// order, coalesced.  No sort, no hash probing, no reduction in global memory.
// The bitmap is cleared through the output columns, so a row's cost does not
// grow with the bitmap: only the unit counters (1/64 of the column count in
// bytes) are swept.
//
// What bounds it: shared memory.  A product costs about 45 shared-memory
// wavefronts per 32 lanes (mark, rank, store, output), and the bitmap's n / 8
// bytes decide how many rows an SM works on.  Measured on one B200 against
// the hash / expand-sort-compress group rows, whose radix sort took half of
// their time (numeric phase, FP64, before -> after): Poisson(25) squares of
// order 20k 0.474 -> 0.197 ms, 200k 4.74 -> 1.86 ms, 600k 15.6 -> 12.6 ms;
// R-MAT of order 20k (8 draws a row) 1.45 -> 0.59 ms, 131k (4) 3.45 -> 1.49
// ms, 400k (2) 6.51 -> 2.95 ms.  Symbolic phase: 0.189 -> 0.128, 1.56 -> 0.75,
// 0.503 -> 0.204, 0.935 -> 0.857 and 1.80 -> 1.28 ms.  Measured and dropped:
// loading the next row's A entries and B row bounds a row ahead (numeric +18 %:
// the registers spill, and the rows of other CTAs already hide the loads), and
// walking rows of long B rows by sub-groups, entry by entry, instead of by the
// flat product number (R-MAT of order 20k symbolic +50 %).
#pragma once

#include "spgemm_cluster.cuh"

namespace tspg {

// Shared-memory layout of a span row for matrices of up to `ncols` columns.
struct SpanLay {
  int nu8;        // groups of 8 units = ceil(ncols / 1024); bitmap at 0
  uint32_t uc;    // uint16 unit counters
  uint32_t pre;   // staged A entries: first product number, B position, value
  uint32_t bq;
  uint32_t av;
  uint32_t keys;  // output columns and values, `cap` slots
  uint32_t vals;
  uint32_t cap;
  uint32_t bytes;
};

__host__ __device__ inline uint32_t span_align(uint32_t x) { return (x + 15u) & ~15u; }

template <int NT, bool NUM, typename PT, typename VT>
__host__ __device__ inline SpanLay span_layout(int64_t ncols, uint32_t cap) {
  SpanLay L;
  L.nu8 = int((ncols + 1023) >> 10);
  L.uc = uint32_t(L.nu8) * 128u;
  L.pre = L.uc + (NUM ? uint32_t(L.nu8) * 16u : 0u);
  L.bq = L.pre + span_align(NT * 4u);
  L.av = L.bq + span_align(NT * uint32_t(sizeof(PT)));
  L.keys = L.av + (NUM ? span_align(NT * uint32_t(sizeof(VT))) : 0u);
  L.vals = L.keys + (NUM ? span_align(cap * 4u) : 0u);
  L.cap = cap;
  L.bytes = L.vals + (NUM ? span_align(cap * uint32_t(sizeof(VT))) : 0u);
  return L;
}

// Most output slots that fit `bytes` of shared memory (0: not even one).
template <int NT, typename PT, typename VT>
__host__ __device__ inline uint32_t span_cap(int64_t ncols, uint32_t bytes) {
  const uint32_t fixed = span_layout<NT, true, PT, VT>(ncols, 0).bytes + 32u;
  if (fixed >= bytes) return 0;
  const uint32_t c = (bytes - fixed) / uint32_t(4 + sizeof(VT));
  return c < 65535u ? c : 65535u;  // unit bases are uint16
}

constexpr int kSpanChunk = 8;  // rows fetched per counter atomic

template <int NT>
struct SpanShared {
  uint32_t len[NT / 32], nz[NT / 32];
  int unit[NT / 32];
  int total;
  unsigned long long slot;
  RowMeta meta[kSpanChunk];
};

// Sums over the warps below warp w (in *below) and over all (in *all) of one
// value per warp left in tmp.
template <int NT, typename T>
__device__ __forceinline__ void span_warp_base(const T *tmp, int w, int lane, T *below, T *all) {
  constexpr int NW = NT / 32;
  if constexpr (NW <= 8) {
    T b = 0, a = 0;
#pragma unroll
    for (int i = 0; i < NW; ++i) {
      const T v = tmp[i];
      if (i < w) b += v;
      a += v;
    }
    *below = b;
    *all = a;
  } else {
    const T x = lane < NW ? tmp[lane] : T(0);
    const T xi = warp_scan_incl(x);
    *below = __shfl_sync(0xffffffffu, xi - x, w);
    *all = __shfl_sync(0xffffffffu, xi, 31);
  }
}

// Stage the A entries [a0, a0 + nc) (nc <= NT) that have products, in order:
// pre = number of the entry's first product, bq = its B row's position minus
// pre (position of product p = bq + p), av = its value.  Ends on a barrier;
// *ne = staged entries, *tot = their products.
template <int NT, bool NUM, typename PT, typename VT>
__device__ __forceinline__ void span_stage(const ProdDev<PT, VT> &P, int64_t a0, int nc,
                                           unsigned char *smem, const SpanLay &L,
                                           SpanShared<NT> &sh, int *ne, uint32_t *tot) {
  using IX = std::conditional_t<sizeof(PT) == 4, uint32_t, int64_t>;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  uint32_t len = 0;
  IX b0 = 0;
  VT a = VT(0);
  if (tid < nc) {
    const int64_t k = __ldg(P.Aj + a0 + tid);
    if constexpr (NUM) a = __ldg(P.Ax + a0 + tid);
    b0 = IX(__ldg(P.Bp + k));
    len = uint32_t(IX(__ldg(P.Bp + k + 1)) - b0);
  }
  const unsigned nzm = __ballot_sync(0xffffffffu, len > 0);
  const uint32_t inc = warp_scan_incl(len);
  if (lane == 31) sh.len[w] = inc;
  if (lane == 0) sh.nz[w] = __popc(nzm);
  __syncthreads();
  uint32_t lb, nb, nall;
  span_warp_base<NT, uint32_t>(sh.len, w, lane, &lb, tot);
  span_warp_base<NT, uint32_t>(sh.nz, w, lane, &nb, &nall);
  if (len > 0) {
    const uint32_t i = nb + __popc(nzm & ((1u << lane) - 1u)), p = lb + inc - len;
    ((uint32_t *)(smem + L.pre))[i] = p;
    ((IX *)(smem + L.bq))[i] = b0 - IX(p);
    if constexpr (NUM) ((VT *)(smem + L.av))[i] = a;
  }
  *ne = int(nall);
  __syncthreads();
}

// Products [t0, t0 + 128) of the staged entries: lane l takes products
// t0 + 32 u + l.  The entry of the first product comes from a warp-wide
// search (two ballots); inside a 32-product window every entry start sets a
// bit of a warp-uniform mask, so a lane's entry is a popcount away.
template <bool NUM, typename IX, typename VT>
__device__ __forceinline__ void span_tile(const uint32_t *pre, const IX *bq, const VT *av, int ne,
                                          uint32_t tot, uint32_t t0,
                                          const int32_t *__restrict__ Bj,
                                          const VT *__restrict__ Bx, int lane, int32_t (&cc)[4],
                                          VT (&vv)[4]) {
  constexpr unsigned FULL = 0xffffffffu;
  const unsigned lt = (1u << lane) - 1u;
  int cur;  // the last entry that starts at or before the window
  if (ne <= 32) {
    cur = __popc(__ballot_sync(FULL, lane < ne && pre[lane] <= t0)) - 1;
  } else {
    const int step = (ne + 31) >> 5, i1 = lane * step;
    const int blk = (__popc(__ballot_sync(FULL, i1 < ne && pre[i1] <= t0)) - 1) * step;
    const int i2 = blk + lane;
    cur = blk + __popc(__ballot_sync(FULL, lane < step && i2 < ne && pre[i2] <= t0)) - 1;
  }
  uint32_t nx = cur + 1 + lane < ne ? pre[cur + 1 + lane] : UINT32_MAX;
  if (__shfl_sync(FULL, nx, 0) >= t0 + 128u) {  // one B row covers the tile
    const IX q0 = bq[cur] + IX(t0 + lane);
    const int32_t *__restrict__ bj = Bj + q0;
    VT a = VT(0);
    if constexpr (NUM) a = av[cur];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const bool in = t0 + 32u * u + lane < tot;
      cc[u] = in ? __ldg(bj + 32 * u) : -1;
      if constexpr (NUM) vv[u] = in ? a * __ldg(Bx + q0 + 32 * u) : VT(0);
    }
    return;
  }
  // more than 32 entries start in the tile: reload them per window
  const bool again = __shfl_sync(FULL, nx, 31) <= t0 + 128u;
  VT xv[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const uint32_t pw = t0 + 32u * u;
    const uint32_t d = nx - (pw + 1u);  // entries starting in (pw, pw + 32]
    const unsigned m = __reduce_or_sync(FULL, d < 32u ? 1u << d : 0u);
    const int j = cur + __popc(m & lt);
    const uint32_t p = pw + lane;
    const IX q = bq[j] + IX(p);
    cc[u] = p < tot ? __ldg(Bj + q) : -1;
    if constexpr (NUM) {
      xv[u] = p < tot ? __ldg(Bx + q) : VT(0);
      vv[u] = av[j];
    }
    cur += __popc(m);
    if (again && u < 3) nx = cur + 1 + lane < ne ? pre[cur + 1 + lane] : UINT32_MAX;
  }
  if constexpr (NUM) {
#pragma unroll
    for (int u = 0; u < 4; ++u) vv[u] *= xv[u];
  }
}

// One row.  NUM: the row's columns and values go to C (m.c slots known, at
// most L.cap).  !NUM: the number of its distinct columns goes to rowc.
// Rows of at most TILES x 4 products per thread (and at most NT A entries)
// keep their products in registers; longer ones walk them twice.  WIPE: the
// bitmap may hold anything on entry (it is cleared here); otherwise it is
// all zero on entry and on return.  save (!NUM): where the bitmap of a row
// that walks its products twice is kept for the numeric phase.  Entered and left with the CTA in step.
template <int NT, bool NUM, int TILES, bool WIPE, typename PT, typename VT>
__device__ __forceinline__ void span_row(const ProdDev<PT, VT> &P, const PhaseArgs &A,
                                         const RowMeta &m, unsigned char *smem, const SpanLay &L,
                                         SpanShared<NT> &sh, uint32_t *save = nullptr) {
  using IX = std::conditional_t<sizeof(PT) == 4, uint32_t, int64_t>;
  constexpr int NW = NT / 32, TP = 128;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  uint32_t *bm = (uint32_t *)smem;
  uint32_t *uc = (uint32_t *)(smem + L.uc);
  const uint32_t *pre = (const uint32_t *)(smem + L.pre);
  const IX *bq = (const IX *)(smem + L.bq);
  const VT *av = (const VT *)(smem + L.av);
  int32_t *keys = (int32_t *)(smem + L.keys);
  VT *vals = (VT *)(smem + L.vals);
  const int nu8 = int((P.n + 1023) >> 10);
  const int64_t a0 = m.a0, na = m.a1 - a0;
  const int32_t *__restrict__ Bj = P.Bj;
  const VT *__restrict__ Bx = P.Bx;
  const bool reg = na <= NT && m.f <= int64_t(TILES) * TP * NW && !P.Ej;
  // entries staged at a time: product numbers inside a stage are 32-bit, so a
  // row of 2^31 products or more (B rows with repeated columns) takes one
  const int64_t step = m.f < (int64_t(1) << 31) ? NT : 1;
  if (WIPE) {
    uint4 *b4 = (uint4 *)smem;
    for (int i = tid; i < nu8 * 8; i += NT) b4[i] = make_uint4(0, 0, 0, 0);
    if (NUM)
      for (int i = tid; i < nu8; i += NT) ((uint4 *)uc)[i] = make_uint4(0, 0, 0, 0);
  }
  if (NUM && !reg)
    for (int64_t e = tid; e < m.c; e += NT) vals[e] = VT(0);
  if (!NUM && tid == 0) sh.total = 0;
  int cnt = 0;
  // true when the product set its column's bit
  auto mark = [&](int32_t col) {
    if constexpr (NUM) return span_mark(bm, uc, uint32_t(col));
    uint32_t *x = bm + (col >> 5);
    const uint32_t bit = 1u << (col & 31);
    if (*(volatile uint32_t *)x & bit) return false;
    if (atomicOr(x, bit) & bit) return false;
    ++cnt;
    return true;
  };
  auto rank_of = [&](int32_t col) { return span_rank(bm, uc, uint32_t(col)); };
  int ne = 0;
  uint32_t tot = 0;
  int32_t cc[TILES][4];
  VT vv[TILES][4];
  unsigned first = 0;
  // the products of TILES tiles of this warp from `base` on, all loads in flight
  auto tiles = [&](auto num, uint32_t base) {
#pragma unroll
    for (int t = 0; t < TILES; ++t) {
      const uint32_t t0 = base + uint32_t(t * NW) * TP;
#pragma unroll
      for (int u = 0; u < 4; ++u) cc[t][u] = -1;
      if (t0 < tot)
        span_tile<decltype(num)::value, IX, VT>(pre, bq, av, ne, tot, t0, Bj, Bx, lane, cc[t],
                                                vv[t]);
    }
  };
  if (reg) {
    span_stage<NT, NUM, PT, VT>(P, a0, int(na), smem, L, sh, &ne, &tot);
    tiles(std::bool_constant<NUM>{}, uint32_t(w) * TP);
#pragma unroll
    for (int t = 0; t < TILES; ++t)
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (cc[t][u] >= 0 && mark(cc[t][u])) first |= 1u << (t * 4 + u);
  } else {
    for (int64_t c0 = 0; c0 < na; c0 += step) {
      span_stage<NT, NUM, PT, VT>(P, a0 + c0, int(min(step, na - c0)), smem, L, sh, &ne, &tot);
      for (uint32_t t0 = uint32_t(w) * TP; t0 < tot; t0 += uint32_t(NW * TILES) * TP) {
        tiles(std::false_type{}, t0);
#pragma unroll
        for (int t = 0; t < TILES; ++t)
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (cc[t][u] >= 0) mark(cc[t][u]);
      }
    }
    if (WIPE || P.Ej) {
      if (na == 0) __syncthreads();  // no staging barrier since the clear
      for_addend<false>(P, m.r, tid, NT, [&](int32_t col, VT) { mark(col); });
    }
  }
  if constexpr (!NUM) {
    cnt = __reduce_add_sync(0xffffffffu, cnt);
    __syncthreads();  // all bits set
    if (lane == 0 && cnt) atomicAdd(&sh.total, cnt);
    if (!WIPE) {
      if (reg) {
#pragma unroll
        for (int t = 0; t < TILES; ++t)
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (cc[t][u] >= 0) bm[cc[t][u] >> 5] = 0u;
      } else {
        for (int i = tid; i < nu8 * 8; i += NT) {
          if (save) ((uint4 *)save)[i] = ((uint4 *)smem)[i];
          ((uint4 *)smem)[i] = make_uint4(0, 0, 0, 0);
        }
      }
    }
    __syncthreads();
    if (tid == 0) {
      A.rowc[m.g] = sh.total;
      if (save && !reg) A.slot[m.g] = int32_t((save - A.bits) / A.slot_words);
    }
    return;
  } else {
    __syncthreads();  // all bits and unit counts set
    // unit counts -> unit bases (thread t owns consecutive groups of 8 units)
    const int per = (nu8 + NT - 1) / NT;
    const int i0 = tid * per, i1 = min(nu8, i0 + per);
    uint4 *u4 = (uint4 *)uc;
    int s = 0;
    for (int i = i0; i < i1; ++i) {
      const uint4 x = u4[i];
      // counts stay below 2^16 in sum: at most 128 per unit, 4 units per half
      const uint32_t y = x.x + x.y + x.z + x.w;
      s += int((y & 0xffffu) + (y >> 16));
    }
    const int inc = warp_scan_incl(s);
    if (lane == 31) sh.unit[w] = inc;
    __syncthreads();
    int below, total;
    span_warp_base<NT, int>(sh.unit, w, lane, &below, &total);
    uint32_t run = uint32_t(below + inc - s);
    for (int i = i0; i < i1; ++i) {
      uint4 x = u4[i];
      uint32_t *h = (uint32_t *)&x;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const uint32_t lo = h[k] & 0xffffu, hi = h[k] >> 16;
        h[k] = (run & 0xffffu) | ((run + lo) << 16);
        run += lo + hi;
      }
      u4[i] = x;
    }
    __syncthreads();
    const int c = int(m.c);
    const bool ok = total == c;  // uniform; false only if the pattern changed
    if (!ok) {
      if (tid == 0) set_error(A.err, 110);
    } else if (reg) {
#pragma unroll
      for (int t = 0; t < TILES; ++t)
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if ((first >> (t * 4 + u)) & 1u) {
            const int r = rank_of(cc[t][u]);
            keys[r] = cc[t][u];
            vals[r] = vv[t][u];
          }
      __syncthreads();
      if (m.f != m.c) {  // the products whose column was marked before them
#pragma unroll
        for (int t = 0; t < TILES; ++t)
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (cc[t][u] >= 0 && !((first >> (t * 4 + u)) & 1u))
              atomicAdd(vals + rank_of(cc[t][u]), vv[t][u]);
        __syncthreads();
      }
    } else {
      auto put = [&](int32_t col, VT v) {
        const int r = rank_of(col);
        keys[r] = col;
        atomicAdd(vals + r, v);
      };
      for (int64_t c0 = 0; c0 < na; c0 += step) {
        if (na > step)
          span_stage<NT, NUM, PT, VT>(P, a0 + c0, int(min(step, na - c0)), smem, L, sh, &ne, &tot);
        for (uint32_t t0 = uint32_t(w) * TP; t0 < tot; t0 += uint32_t(NW * TILES) * TP) {
          tiles(std::bool_constant<NUM>{}, t0);
#pragma unroll
          for (int t = 0; t < TILES; ++t)
#pragma unroll
            for (int u = 0; u < 4; ++u)
              if (cc[t][u] >= 0) put(cc[t][u], vv[t][u]);
        }
      }
      for_addend<true>(P, m.r, tid, NT, put);
      __syncthreads();
    }
    if (ok) {
      int32_t *__restrict__ Cj = P.Cj + m.off;
      VT *__restrict__ Cx = P.Cx + m.off;
      for (int e = tid; e < c; e += NT) {
        const int32_t k = keys[e];
        Cj[e] = k;
        Cx[e] = vals[e];
        if (!WIPE) bm[k >> 5] = 0u;
      }
    } else if (!WIPE) {
      for (int i = tid; i < nu8 * 8; i += NT) ((uint4 *)smem)[i] = make_uint4(0, 0, 0, 0);
    }
    if (!WIPE)
      for (int i = tid; i < nu8; i += NT) u4[i] = make_uint4(0, 0, 0, 0);
    __syncthreads();
  }
}

// The rows of classes [c0, c1) (contiguous lists) as span rows, persistent:
// CTAs of NT threads (several per SM, as the layout allows) take chunks of
// rows from the counter of class c0.
template <int NT, bool NUM, typename PT, typename VT>
__global__ void __launch_bounds__(NT, 1024 / NT)
    k_span(const ProdDev<PT, VT> *prods, PhaseArgs A, SpanLay L, int c0, int c1) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ SpanShared<NT> sh;
  const int tid = threadIdx.x;
  phase_begin();
  int64_t count = 0;
  for (int c = c0; c < c1; ++c) count += A.S->cnt[c];
  const int64_t base = A.S->off[c0];
  if (count == 0) {
    phase_end();
    return;
  }
  for (int i = tid; i < L.nu8 * (NUM ? 9 : 8); i += NT)
    ((uint4 *)smem)[i] = make_uint4(0, 0, 0, 0);  // bitmap, then unit counters
  while (true) {
    if (tid == 0) {
      const unsigned long long cur = *(volatile unsigned long long *)&A.S->next[c0];
      const int64_t left = count - int64_t(cur);
      const unsigned long long take = left > int64_t(kSpanChunk) * gridDim.x * 2 ? kSpanChunk : 1ull;
      sh.slot = atomicAdd(&A.S->next[c0], take) | (take << 48);
    }
    __syncthreads();
    const unsigned long long v = sh.slot;
    const int64_t i0 = int64_t(v & ((1ull << 48) - 1));
    if (i0 >= count) break;
    const int nrow = int(min(count - i0, int64_t(v >> 48)));
    if (tid < nrow) sh.meta[tid] = load_meta<NUM>(prods, A, base + i0 + tid);
    __syncthreads();
    for (int t = 0; t < nrow; ++t) {
      const long long t0 = clock64();
      const RowMeta m = sh.meta[t];
      uint32_t *save = nullptr;  // the first rows of the DENSE classes have slots
      if (!NUM && c0 == 0 && A.bits && i0 + t < A.nslots) save = A.bits + (i0 + t) * A.slot_words;
      span_row<NT, NUM, NUM ? 2 : 4, false, PT, VT>(prods[m.p], A, m, smem, L, sh, save);
      if (A.prof) {
        int c = c0;
        while (c + 1 < c1 && base + i0 + t >= A.S->off[c + 1]) ++c;
        prof_add(A, c, t0, tid == 0);
      }
    }
  }
  phase_end();
}

// The numeric DENSE rows of the rank form (at most kRankMaxCols columns, not
// taken by the column-window rule), persistent, before k_phase: 24 or 32 warps
// per SM (one CTA of 768 threads or two of 512), where k_phase's 16 warps keep
// the 128 registers of the hash rows' radix sort.  Rows whose output fits the
// CTA's `bytes` of shared memory beside the bitmap are span rows.  Heavy rows (DENSE0 / DENSE1) are spread over the DENSE2 rows
// as in k_phase, so few of their reduction targets are live at once.
template <int NT, int CT, typename PT, typename VT>
__global__ void __launch_bounds__(NT, CT)
    k_dense_rank(const ProdDev<PT, VT> *prods, PhaseArgs A, uint32_t bytes) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ PhaseShared sh;
  __shared__ SpanShared<NT> ss;
  __shared__ unsigned long long s_item;
  const int tid = threadIdx.x;
  phase_begin();
  const int64_t H = A.S->cnt[CLS_DENSE0] + A.S->cnt[CLS_DENSE1];
  const int64_t L = A.S->cnt[CLS_DENSE2];
  const int64_t c01 = A.S->cnt[CLS_DENSE0];
  const int64_t K = H > 0 ? min(int64_t(kHeavyPeriod), 1 + L / H) : 1;
  GroupMem gm;
  gm.cnt = nullptr;
  gm.tmp = sh.scan;
  gm.itmp = sh.itmp;
  gm.lst = sh.lst;
  gm.nl = sh.nl + 47;
  gm.cap = 1024;
  gm.stage = nullptr;
  while (true) {
    if (tid == 0) s_item = atomicAdd(&A.S->work3, 1ull);
    __syncthreads();
    const int64_t item = (int64_t)s_item;
    __syncthreads();
    if (item >= H + L) break;
    int64_t pos = item;
    if (K > 1 && item < K * H) pos = item % K == 0 ? item / K : H + (item - item / K - 1);
    // the DENSE classes' lists are contiguous: DENSE0, DENSE1, DENSE2
    const int c = pos < c01 ? CLS_DENSE0 : pos < H ? CLS_DENSE1 : CLS_DENSE2;
    const int64_t idx = A.S->off[CLS_DENSE0] + pos;
    const long long t0 = clock64();
    const RowRef rr = decode_row(A, idx);
    const ProdDev<PT, VT> &P = prods[rr.p];
    const int64_t c_row = A.rowc[rr.g];
    const uint32_t cap = P.n <= kRankMaxCols
                             ? span_cap<NT, PT, VT>(P.n, bytes) : 0;
    if (c_row <= int64_t(cap) && P.n <= kRankMaxCols &&
        !win_row(P, A.rowf[rr.g], c_row, A.S->tune)) {
      const SpanLay L = span_layout<NT, true, PT, VT>(P.n, cap);
      const RowMeta m = load_meta<true>(prods, A, idx);
      span_row<NT, true, (NT > 512 ? 2 : 1), true, PT, VT>(P, A, m, smem, L, ss);
      prof_add(A, c, t0, tid == 0);
    } else if (P.n <= kRankMaxCols && !win_row(P, A.rowf[rr.g], int64_t(A.rowc[rr.g]), A.S->tune)) {
      num_dense_rank_row<NT, PT, VT>(prods, A, idx, smem, gm);
      prof_add(A, c, t0, tid == 0);
    } else if (tid == 0) {
      A.S->rank_left = 1;  // read by k_phase, which runs after this kernel
    }
    __syncthreads();
  }
  phase_end();
}

// Two CTAs of k_dense_rank per SM when every rank row fits half of its shared
// memory: one row's bitmap and emission passes run while another's value pass
// waits on the L2's reductions (R-MAT of order 2^18, 16 draws a row: 27.7 ->
// 23.9 ms).  Fewer rows than a few per SM end on the longest one, which the
// 768-thread CTA finishes sooner (order 30k, 138 rows: 0.44 against 0.20 ms).
constexpr uint32_t kRank2Smem = 100 * 1024;
constexpr int kRank2Rows = 8;  // DENSE rows per SM
constexpr uint32_t kSpanSmemMax = 220 * 1024;  // dynamic; the static part stays below 7 KiB

// CTAs of k_span resident on one SM with this layout (64 registers a thread).
template <int NT>
inline int span_ctas(const SpanLay &L) {
  if (L.bytes > kSpanSmemMax) return 0;
  const uint32_t per = L.bytes + uint32_t(sizeof(SpanShared<NT>)) + 1024u;
  const int by_smem = int((228u * 1024u) / per), by_regs = 1024 / NT;
  return by_smem < by_regs ? by_smem : by_regs;
}

template <int NT, bool NUM, typename PT, typename VT>
inline cudaError_t launch_span(tspg_ctx *ctx, cudaStream_t s, const ProdDev<PT, VT> *prods,
                               const PhaseArgs &pa, const SpanLay &L, int c0, int c1,
                               bool overlap) {
  const int ctas = span_ctas<NT>(L);
  ctx->launches += 1;
  return launch_phase(overlap, ctx->num_sms * ctas, NT, L.bytes, s, k_span<NT, NUM, PT, VT>, prods,
                      pa, L, c0, c1);
}

// Sorted B rows only matter to rows swept in column windows: wider than the
// rank form's bitmap, or taken by the window form of the tuning.
inline bool needs_sorted(const Tune &t, int64_t ncols) { return ncols > kRankMaxCols || t.win != 0; }

// The row binning of a run: the caller's, where a bound at its default (the
// table's capacity) leaves the choice to the width.  While the bitmap of 128-thread span rows stays
// small (8 CTAs per SM), numeric rows of more than kSpanWarpRow outputs leave
// the warps for them.  Uniform rows of order 1024 with ~250 outputs: numeric
// 49 -> 15 us; Poisson(15) of order 100k (~225 outputs) 0.55 -> 0.48 ms, of
// order 200k (5 CTAs per SM) 1.16 -> 1.23 ms; ~144 outputs, order 120k 0.56 ->
// 0.60 ms.  And where 512-thread span rows with the full
// bound's slots would have an SM to themselves, the bound drops to
// kSpanHalfRow, at which two fit, the longer rows going to the DENSE kernel:
// R-MAT of order 65k 1.39 -> 1.21 ms, 131k 2.05 -> 1.90 ms (a whole call); of
// order 30k, where two fit anyway, 0.78 -> 0.83 ms.
constexpr int64_t kSpanWarpCols = 131072;
constexpr int32_t kSpanWarpRow = 192;
constexpr int32_t kSpanHalfRow = 4096;
template <typename PT, typename VT>
inline Tune span_tune(Tune t, int64_t ncols, bool addend) {
  t.lane = addend ? 0 : kLaneSlots;  // lane rows take no addend
  if (ncols <= kSpanWarpCols && t.num[0] == kNumLim32 && t.num[1] >= t.num[0])
    t.num[0] = kSpanWarpRow;
  if (t.num[3] == kNumLim1024 && t.num[2] <= kSpanHalfRow && ncols <= kRankMaxCols &&
      span_ctas<512>(span_layout<512, true, PT, VT>(ncols, uint32_t(t.num[3]))) < 2 &&
      span_ctas<512>(span_layout<512, true, PT, VT>(ncols, uint32_t(kSpanHalfRow))) >= 2)
    t.num[3] = kSpanHalfRow;
  return t;
}

// A class takes the span form when at least two of its CTAs fit an SM: with
// one, too few rows are in flight (numeric, R-MAT of order 800k: 9.44 ms as
// span rows at one CTA per SM, 8.77 ms as hash rows; symbolic at two: 2.38
// against 3.85 ms).  The numeric 512-thread rows replace rows that had an SM
// to themselves, so one CTA is enough for them.
//
// The symbolic DENSE and G1024 rows are span rows (which can keep their bitmaps)
// up to this width.
template <typename PT, typename VT>
inline bool sym_dense_span(int64_t ncols) {
  return span_ctas<512>(span_layout<512, false, PT, VT>(ncols, 0)) >= 2;
}

// The persistent kernels of a symbolic phase (one-pass rows aside).
template <typename PT, typename VT>
inline int launch_symbolic_rows(tspg_ctx *ctx, cudaStream_t s, const ProdDev<PT, VT> *prods,
                                PhaseArgs pa, int64_t ncols, bool may_overlap) {
  const SpanLay L1 = span_layout<128, false, PT, VT>(ncols, 0);
  const SpanLay L2 = span_layout<256, false, PT, VT>(ncols, 0);
  const SpanLay L3 = span_layout<512, false, PT, VT>(ncols, 0);
  if (sym_dense_span<PT, VT>(ncols)) {
    TSPG_CUDA(ctx, (launch_span<512, false, PT, VT>(ctx, s, prods, pa, L3, 0, CLS_G1024 + 1, false)));
  } else {
    k_phase<PT, VT, false><<<ctx->num_sms, kSymThreads, kDynSmem, s>>>(prods, pa);
    ctx->launches += 1;
  }
  const bool overlap = may_overlap && sym_dense_span<PT, VT>(ncols);  // k_phase lets nothing start early
  if (span_ctas<256>(L2) >= 2) {
    TSPG_CUDA(ctx, (launch_span<256, false, PT, VT>(ctx, s, prods, pa, L2, CLS_G256, CLS_G256 + 1,
                                                    overlap)));
    pa.skip |= 1u << CLS_G256;
  }
  if (span_ctas<128>(L1) >= 2) {
    TSPG_CUDA(ctx, (launch_span<128, false, PT, VT>(ctx, s, prods, pa, L1, CLS_G128, CLS_G128 + 1,
                                                    overlap)));
    pa.skip |= 1u << CLS_G128;
  }
  TSPG_CUDA(ctx, launch_phase(overlap, ctx->num_sms, kGroupThreads, kGroupDynSmem, s,
                              k_groups<PT, VT, false>, prods, pa));
  ctx->launches += 1;
  return TSPG_OK;
}

// One numeric class of `rows` rows (-1: not known) with at most `cap` outputs
// each, as span rows of NT threads; a class too small to give every SM its
// CTAs takes wider ones, so that its last row ends sooner.
template <int NT, typename PT, typename VT>
inline cudaError_t launch_span_class(tspg_ctx *ctx, cudaStream_t s,
                                     const ProdDev<PT, VT> *prods, const PhaseArgs &pa,
                                     int64_t ncols, uint32_t cap, int cls, int64_t rows,
                                     bool overlap) {
  if constexpr (NT < 512) {
    if (rows >= 0 && rows <= int64_t(ctx->num_sms) * (512 / NT))
      return launch_span_class<2 * NT, PT, VT>(ctx, s, prods, pa, ncols, cap, cls, rows, overlap);
  }
  return launch_span<NT, true, PT, VT>(ctx, s, prods, pa,
                                       span_layout<NT, true, PT, VT>(ncols, cap), cls, cls + 1,
                                       overlap);
}

// Products an output from which a class of many rows (a row or a few for every
// SM) takes the hash form instead of the span form, which walks the products
// twice.  Numeric phase, hash and span: 5,000 rows of 20,000 products on 400
// columns 0.54 and 0.70 ms; 1,000 of 200,000 on 2,000 1.18 and 1.33; 300 of
// 800,000 on 4,000 1.39 and 2.26; at 20 products an output (5,000 rows on 2,000
// columns) 1.25 and 1.13.  Fewer rows than that end on the longest one, which
// the wider span rows finish sooner (200 of 100,000 on 500: 0.42 and 0.23 ms).
constexpr int64_t kHashPerOut = 24;
// The persistent kernels of a numeric phase whose products have at most
// `ncols` columns; tn: the run's row binning (span_tune), the one in its Sched
// records, by which the rows were classed: a kept plan runs with the tuning of
// its symbolic call, whatever the context's is by now.  cnt: rows per class
// when the host knows them (else null).
// per_out: products an output of the run (0: not known).  skip_empty: no kernel
// is launched for an empty class (small products, where a launch counts).
template <typename PT, typename VT>
inline int launch_numeric_rows(tspg_ctx *ctx, cudaStream_t s, const ProdDev<PT, VT> *prods,
                               PhaseArgs pa, int64_t ncols, const Tune &tn, const int64_t *cnt,
                               int64_t per_out, bool skip_empty, bool may_overlap) {
  TSPG_CUDA(ctx, launch_dense_cluster<PT, VT>(ctx, s, prods, pa, tn.cluster));
  auto rows = [&](int c) { return cnt ? cnt[c] : int64_t(-1); };
  auto some = [&](int c) { return !skip_empty || rows(c) != 0; };
  // many rows of many products an output: the hash forms, which walk them once
  auto hashed = [&](int c, int per_sm) {
    return per_out >= kHashPerOut && rows(c) >= int64_t(per_sm) * ctx->num_sms;
  };
  const int64_t dense = cnt ? cnt[CLS_DENSE0] + cnt[CLS_DENSE1] + cnt[CLS_DENSE2] : -1;
  const uint32_t nb = uint32_t((ncols + 1023) >> 10);
  bool overlap = false;  // the first kernel of the phase starts after the binning
  if (!skip_empty || dense != 0) {
    if (nb * 196u <= kRank2Smem && dense >= int64_t(kRank2Rows) * ctx->num_sms)
      TSPG_CUDA(ctx, launch_phase(overlap, ctx->num_sms * 2, 512, kRank2Smem, s,
                                  k_dense_rank<512, 2, PT, VT>, prods, pa, kRank2Smem));
    else
      TSPG_CUDA(ctx, launch_phase(overlap, ctx->num_sms, kRankThreads, kDynSmem, s,
                                  k_dense_rank<kRankThreads, 1, PT, VT>, prods, pa,
                                  uint32_t(kDynSmem)));
    ctx->launches += 1;
    overlap = may_overlap;
  }
  if (!hashed(CLS_G1024, 1) && span_ctas<512>(span_layout<512, true, PT, VT>(ncols, uint32_t(tn.num[3]))) >= 1) {
    pa.skip |= 1u << CLS_G1024;
    if (some(CLS_G1024)) {
      TSPG_CUDA(ctx, (launch_span_class<512>(ctx, s, prods, pa, ncols, uint32_t(tn.num[3]),
                                             CLS_G1024, rows(CLS_G1024), overlap)));
      overlap = may_overlap;
    }
  }
  if (!hashed(CLS_G256, 3) && span_ctas<256>(span_layout<256, true, PT, VT>(ncols, uint32_t(tn.num[2]))) >= 2) {
    pa.skip |= 1u << CLS_G256;
    if (some(CLS_G256)) {
      TSPG_CUDA(ctx, (launch_span_class<256>(ctx, s, prods, pa, ncols, uint32_t(tn.num[2]),
                                             CLS_G256, rows(CLS_G256), overlap)));
      overlap = may_overlap;
    }
  }
  if (!hashed(CLS_G128, 6) && span_ctas<128>(span_layout<128, true, PT, VT>(ncols, uint32_t(tn.num[1]))) >= 2) {
    pa.skip |= 1u << CLS_G128;
    if (some(CLS_G128)) {
      TSPG_CUDA(ctx, (launch_span_class<128>(ctx, s, prods, pa, ncols, uint32_t(tn.num[1]),
                                             CLS_G128, rows(CLS_G128), overlap)));
      overlap = may_overlap;
    }
  }
  // k_phase: DENSE rows that are neither rank nor span rows, G1024 hash rows
  const bool left = ncols > kRankMaxCols || tn.win != 0;
  if ((left && (!skip_empty || dense != 0)) ||
      (!(pa.skip >> CLS_G1024 & 1u) && some(CLS_G1024))) {
    k_phase<PT, VT, true><<<ctx->num_sms, kThreads, kDynSmem, s>>>(prods, pa);  // reads rank_left
    ctx->launches += 1;
    overlap = false;
  }
  if (some(CLS_LANE)) {
    TSPG_CUDA(ctx, launch_phase(overlap, ctx->num_sms, kOnepassThreads, kOnepassSmem, s,
                                k_lanes<true, PT, VT>, prods, pa));
    ctx->launches += 1;
    overlap = may_overlap;
  }
  if (some(CLS_G32) || (!(pa.skip >> CLS_G256 & 1u) && some(CLS_G256)) ||
      (!(pa.skip >> CLS_G128 & 1u) && some(CLS_G128))) {
    TSPG_CUDA(ctx, launch_phase(overlap, ctx->num_sms, kGroupThreads, kGroupDynSmem, s,
                                k_groups<PT, VT, true>, prods, pa));
    ctx->launches += 1;
  }
  TSPG_CUDA(ctx, cudaGetLastError());
  return TSPG_OK;
}

// Dynamic shared-memory limits of the persistent kernels (a per-device
// attribute of each kernel; the caller has made ctx->device current), raised
// once by each context.
template <typename PT, typename VT>
inline int set_smem_attr(tspg_ctx *ctx) {
  const uint32_t mine = 1u << ((sizeof(PT) == 8 ? 2 : 0) + (sizeof(VT) == 8 ? 1 : 0));
  if (ctx->smem_raised & mine) return TSPG_OK;
  auto raise = [](auto *k, int bytes) {
    return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess;
  };
  if (!raise(k_phase<PT, VT, false>, kDynSmem) || !raise(k_phase<PT, VT, true>, kDynSmem) ||
      !raise(k_groups<PT, VT, false>, kGroupDynSmem) ||
      !raise(k_groups<PT, VT, true>, kGroupDynSmem) || !raise(k_lanes<false, PT, VT>, kOnepassSmem) ||
      !raise(k_lanes<true, PT, VT>, kOnepassSmem) ||
      !raise(k_dense_rank<kRankThreads, 1, PT, VT>, kDynSmem) || !raise(k_dense_rank<512, 2, PT, VT>, kRank2Smem) ||
      !raise(k_span<128, false, PT, VT>, kSpanSmemMax) || !raise(k_span<256, false, PT, VT>, kSpanSmemMax) || !raise(k_span<512, false, PT, VT>, kSpanSmemMax) || !raise(k_span<128, true, PT, VT>, kSpanSmemMax) ||
      !raise(k_span<256, true, PT, VT>, kSpanSmemMax) ||
      !raise(k_span<512, true, PT, VT>, kSpanSmemMax))
    return TSPG_ECUDA;
  ctx->smem_raised |= mine;
  return TSPG_OK;
}

}  // namespace tspg
