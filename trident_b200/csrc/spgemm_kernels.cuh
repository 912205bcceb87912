// spgemm_kernels.cuh — device side of the two-phase row-wise SpGEMM.
//
// Layout in HBM.  Operands are plain CSR (row offsets int32 or int64, int32
// column indices, FP64 or FP32 values).  A launch covers one or many products
// ("prods"); rows of all products are numbered globally (row g of product p
// is g = base[p] + r) so that binning, scans and the persistent work queue
// see one flat row space.  Per global row the plan keeps:
//   rowf[g]  int64  products (a.k.a. mults / flops/2) of the row
//   rowc[g]  int32  distinct output columns (symbolic result)
//   cp[g]    int64  exclusive prefix of rowc over the flat row space
//   list[]   uint64 rows binned by class, entry = (p << 40) | r
//
// Row classes (shared by both phases, heaviest first so that the persistent
// grid starts on the long rows).  Where a bitmap of the column range leaves
// room for two CTAs per SM, rows of every class but the shortest take the span
// form instead of the one named here (spgemm_span.cuh):
//   DENSE  (three sub-classes by product count, heaviest first) one CTA per
//          row.  Symbolic: a bitmap of the whole column range in shared
//          memory.  Numeric: the same bitmap, then a CTA scan that writes the
//          sorted columns and keeps a rank base per 32 columns; every product
//          is then added into its output slot with a global FP64 reduction
//          (rows wider than the shared-memory bitmap use an FP64 window of
//          16384 columns swept with per-A-entry cursors instead).
//   G1024  one CTA per row, open-addressing hash in shared memory.
//   G256   256-thread groups, named barriers.
//   G128   128-thread groups.
//   G32    one warp per row.
//   LANE   one lane per row, 32 rows by a warp: numeric rows of at most 27
//          outputs, and the one-pass rows of the symbolic launch.
// Hash rows are sorted after accumulation by an in-place compaction into the
// first half of the table and a stable LSD radix sort (bitonic below 65).
#pragma once

#include "internal.cuh"

namespace tspg {

constexpr int kThreads = 512;   // persistent CTA: 16 warps x 128 registers
// The symbolic CTA rows need no values (64 registers), so their persistent
// CTA runs 32 warps: more B-row loads and bitmap updates in flight per SM
// (R-MAT 20 symbolic phase: 58.4 ms at 16 warps, 49.4 at 24, 46.0 at 32).
constexpr int kSymThreads = 1024;
// The numeric DENSE rows of the rank form (k_dense_rank) likewise: their
// bitmap, scan and emission passes carry no values, and the value pass's
// 8 loads in flight fit 80 registers (8 bytes spilled with int32 offsets
// and FP64 values).  1024 threads (64 registers) measured the same.
constexpr int kRankThreads = 768;
constexpr int kTableSmem = 196608;              // hash tables / dense window
constexpr int kCountSmem = 16384;               // radix-sort digit counters
constexpr int kDynSmem = kTableSmem + kCountSmem;  // one CTA per SM
// The group-row kernel (k_groups): 24 warps x 80 registers over the same
// table space, so more rows are in flight per SM than the 16 warps of the
// persistent CTA-row kernel (group rows are latency-bound: shared-memory
// probes and the loads of short B rows); 1 KiB of digit counters per warp.
constexpr int kGroupThreads = 768;
constexpr int kGroupCountSmem = (kGroupThreads / 32) * 1024;
constexpr int kGroupDynSmem = kTableSmem + kGroupCountSmem;

// Row classes, heaviest first.  The first four are worked by the whole CTA
// (items fetched by one thread); G256 / G128 / G32 rows are fetched by each
// group on its own, so groups never wait for one another.
constexpr int NCLS = 8;
enum {
  CLS_DENSE0 = 0,  // DENSE rows with >= 2^20 products
  CLS_DENSE1 = 1,  // DENSE rows with >= 2^17 products
  CLS_DENSE2 = 2,  // other DENSE rows
  CLS_G1024 = 3,
  CLS_G256 = 4,
  CLS_G128 = 5,
  CLS_G32 = 6,
  CLS_ONEPASS = 7,  // symbolic: rows computed whole in the symbolic launch
  CLS_LANE = 7      // numeric: short rows, 32 of them by one warp, a lane each
};
constexpr int kCtaClasses = 4;  // classes [0, 4) are CTA-level
__host__ __device__ constexpr bool cls_dense(int c) { return c <= CLS_DENSE2; }

constexpr int kSymT32 = 1024, kSymT128 = 4096, kSymT256 = 8192,
              kSymT1024 = 32768;
constexpr int kNumT32 = 512, kNumT128 = 2048, kNumT256 = 4096,
              kNumT1024 = 16384;
constexpr int kDenseW = 16384;           // numeric dense window (columns)
constexpr int kDenseCurSmem = 8192;      // cursors kept in shared memory
constexpr int64_t kDenseBits = int64_t(kTableSmem + kCountSmem) * 8;  // whole-row bitmap
constexpr int kBitonicMax = 64;          // rows up to this size sort bitonic
// whole-row DENSE numeric form: per 32 columns a bitmap word (4 B) and a
// uint16 rank offset, per 1024 columns an int block base (196 B per block)
constexpr int64_t kRankMaxCols = int64_t(kDynSmem / 196) * 1024;
// numeric CTA-level rows: at most one heavy (DENSE0 / DENSE1) row per this
// many items; the period is also capped at 1 + light / heavy rows, so in
// practice the heavy rows spread evenly over the whole item sequence (R-MAT
// 20: 309.9 ms heaviest-first, 299.7 / 292.5 / 289.7 ms with periods 4 / 8 / 11)
constexpr int kHeavyPeriod = 64;

__host__ __device__ inline int dense_sub(int64_t f) {
  return f >= (int64_t(1) << 20) ? CLS_DENSE0 : f >= (int64_t(1) << 17) ? CLS_DENSE1 : CLS_DENSE2;
}
// How a run's totals bear on a row's class (set with the list offsets).
struct RowRule {
  // products above which a warp, 128- or 256-thread row is worked by more threads
  int64_t wide32 = 2048, wide128 = 8192, wide256 = 32768;
  int64_t lane = INT64_MAX;  // ... up to which a row of few outputs is a lane row
};
// A group row by its products: many products on few columns (hub rows of a
// small matrix) take more threads than their table asks for.  R-MAT of order
// 1318 (FP32): 128-thread rows of 10^4 products were the call (0.17 ms).
__host__ __device__ inline int wide_class(int c, int64_t f, const RowRule &r = RowRule()) {
  if (c == CLS_G32 && f > r.wide32) c = CLS_G128;
  if (c == CLS_G128 && f > r.wide128) c = CLS_G256;
  if (c == CLS_G256 && f > r.wide256) c = CLS_G1024;
  return c;
}
// ... in the numeric phase only while the row is more than its share of the
// run's products, so that the others do not cover it: 24, 12 and 6 such groups
// per SM.  70,000 rows of 2,400 products and 150 outputs: warps 1.21 ms, 128
// threads each 1.92; 5,000 rows of 6,080 and 190: 0.29 and 0.38 ms.
//
// Lane rows want 32 rows a warp to be worth it (k_lanes has 16 warps per SM):
// with r rows to a warp they take ~130 issue slots a product of the longest
// row, single warps ~1500 a row and 8 a product.  20,000 rows (8.4 to a warp):
// 144 products 59 us by lanes and 80 by warps, 240 86 and 89, 810 283 and 142.
__device__ inline RowRule row_rule(int64_t products, int64_t rows) {
  constexpr int64_t kSms = 148, kLaneWarps = kSms * 16;
  RowRule r;
  r.wide32 = max(r.wide32, products / (kSms * 24));
  r.wide128 = max(r.wide128, products / (kSms * 12));
  r.wide256 = max(r.wide256, products / (kSms * 6));
  r.lane = rows >= 16 * kLaneWarps ? INT64_MAX : 1500 * rows / (130 * kLaneWarps - 8 * rows);
  return r;
}
__host__ __device__ inline int sym_class(int64_t f, int64_t n, const Tune &t) {
  const int64_t fe = f < n ? f : n;
  if (f == 0) return -1;
  if (fe <= t.sym[0]) return wide_class(CLS_G32, f);
  if (fe <= t.sym[1]) return wide_class(CLS_G128, f);
  if (fe <= t.sym[2]) return wide_class(CLS_G256, f);
  if (fe <= t.sym[3]) return CLS_G1024;
  return dense_sub(f);
}
// One-pass rows (plain products only, Sched::onepass set): rows of the
// symbolic warp, 128- and 256-thread classes are multiplied whole in the
// symbolic launch (k_lanes: a lane per row, or a warp per row where the 32
// rows of a warp are uneven or the row holds more columns than a lane's table);
// their output waits in a scratch buffer for the numeric launch, which copies
// it into C.  A row that turns out to hold more columns than the warp's table
// takes is deferred to the two-pass path — so no row writes more than
// kCappedCols scratch entries, and the scratch stays dense.
constexpr int kCappedCols = 32;
__host__ __device__ inline bool onepass_row(int64_t f, int64_t n, const Tune &t) {
  const int64_t fe = f < n ? f : n;
  return f > 0 && fe <= t.sym[2];
}
// A one-pass row whose whole table fits 64 slots (else only its capped
// 64-slot attempt can finish it), and the scratch entries it may write.
__host__ __device__ inline bool onepass_full(int64_t f, int64_t n, const Tune &t) {
  const int64_t fe = f < n ? f : n;
  return int64_t(t.load) * fe <= 2 * kCappedCols;
}
__host__ __device__ inline int64_t onepass_bound(int64_t f, int64_t n, const Tune &t) {
  const int64_t fe = f < n ? f : n;
  return onepass_full(f, n, t) ? fe : kCappedCols;
}
__host__ __device__ inline int num_class(int64_t c, int64_t f, const Tune &t, const RowRule &r) {
  if (c == 0 || f < 0) return -1;  // f < 0: a one-pass row, already computed
  if (c <= t.lane && f <= r.lane) return CLS_LANE;
  if (c <= t.num[0]) return wide_class(CLS_G32, f, r);
  if (c <= t.num[1]) return wide_class(CLS_G128, f, r);
  if (c <= t.num[2]) return wide_class(CLS_G256, f, r);
  if (c <= t.num[3]) return CLS_G1024;
  return dense_sub(f);
}


template <typename PT, typename VT>
struct ProdDev {
  const PT *Ap;
  const int32_t *Aj;
  const VT *Ax;
  const PT *Bp;
  const int32_t *Bj;
  const VT *Bx;
  int64_t m, n;
  int32_t *Cj;
  VT *Cx;
  void *Cp;       // output rowptr (product-local), cp_bits wide
  int32_t cp_bits;
  int32_t b_sorted;
  int32_t b_strict;  // B's rows were found strictly increasing (k_check_strict)
  // optional addend of C = E + A·B (tspg_spgemm_acc): E's row r joins row r's
  // products as entries with coefficient 1; Ej == nullptr when there is none
  const void *Ep;
  const int32_t *Ej;
  const VT *Ex;
  int32_t ep_bits;
};

template <typename PT, typename VT>
__device__ __forceinline__ void addend_row(const ProdDev<PT, VT> &P, int64_t r, int64_t &e0,
                                           int64_t &e1) {
  if (P.ep_bits == 32) {
    e0 = ((const int32_t *)P.Ep)[r];
    e1 = ((const int32_t *)P.Ep)[r + 1];
  } else {
    e0 = ((const int64_t *)P.Ep)[r];
    e1 = ((const int64_t *)P.Ep)[r + 1];
  }
}

// Work schedule of one phase: rows per class, their list offsets and the
// work-item prefix the persistent kernel decodes.
// A run's numeric record follows its symbolic one in memory.
struct Sched {
  Tune tune;  // row binning of this run, set by k_set_tune after the reset
  int64_t cnt[NCLS];
  int64_t off[NCLS];
  int64_t cur[NCLS];
  unsigned long long next[NCLS];  // per-class row counters of the group-level classes
  unsigned long long work;        // item counter of the CTA-level classes
  int64_t total;      // sum of mults (symbolic) or of nnz (numeric)
  int64_t upper;      // sum of min(mults, ncols)
  int64_t max_a_row;  // longest A row (sizes the DENSE cursor scratch)
  int64_t nonempty;
  unsigned long long work2;  // row counter of the cluster kernel (column-window rows)
  int32_t onepass;  // symbolic record of a plain product: one-pass rows on
  uint32_t ticket;  // blocks done, of the kernel whose last block finishes a step
  int64_t cand[NCLS];           // one-pass candidates by the class they left
  unsigned long long ndefer;    // one-pass rows sent back to the two-pass path
  unsigned long long work3;     // row counter of the rank-form DENSE kernel
  int32_t rank_left;            // DENSE rows that kernel left to k_phase (0 / 1)
  int32_t pad32b;
  unsigned long long nlong;     // A rows left to k_row_mults_long
  RowRule rule;                 // symbolic record: for the numeric classes
};

__device__ __forceinline__ int find_prod(const int64_t *base, int nprod,
                                         int64_t g) {
  int lo = 0, hi = nprod;
  while (hi - lo > 1) {
    int mid = (lo + hi) >> 1;
    if (base[mid] <= g) lo = mid; else hi = mid;
  }
  return lo;
}

__device__ __forceinline__ uint32_t hash_slot(int32_t col, int logT) {
  return ((uint32_t)col * 2654435761u) >> (32 - logT);
}

__device__ __forceinline__ int ilog2_pow2(uint32_t x) { return 31 - __clz(x); }

__device__ __forceinline__ uint32_t pow2_at_least(int64_t x, uint32_t lo) {
  uint32_t t = lo;
  while ((int64_t)t < x) t <<= 1;
  return t;
}

// Sub-group width for the CTA rows' product loop (for_products_balanced):
// threads of a sub-group walk one B row together, sized to the row's average
// B row length f / na.
__device__ __forceinline__ int subgroup_width_avg(int64_t f, int64_t na, int G) {
  int64_t avg = na > 0 ? f / na : 0;
  int S = avg >= 24 ? 32 : avg >= 12 ? 16 : avg >= 6 ? 8 : avg >= 3 ? 4 : 2;
  return S > G ? G : S;
}

// ---------------------------------------------------------------------------
// Setup kernels

// Row binning of a run into its Sched records (after they were zeroed).
static __global__ void k_set_tune(Sched *S, int n, Tune t, int onepass = 0) {
  if (threadIdx.x < n) {
    S[threadIdx.x].tune = t;
    S[threadIdx.x].onepass = threadIdx.x == 0 ? onepass : 0;
  }
}

// Everything a single product's symbolic phase starts from, in one launch of
// one block (two memsets and two kernels before): the Sched records zeroed,
// their row binning, the product's descriptor and row base.
template <typename PT, typename VT>
__global__ void __launch_bounds__(128) k_setup(ProdDev<PT, VT> *dst, ProdDev<PT, VT> v,
                                               int64_t *base, Sched *S, int n, Tune t,
                                               int onepass) {
  uint64_t *w = (uint64_t *)S;
  static_assert(sizeof(Sched) % 8 == 0, "Sched is zeroed by words");
  for (int i = threadIdx.x; i < int(n * sizeof(Sched) / 8); i += blockDim.x) w[i] = 0;
  __syncthreads();
  if (threadIdx.x < n) {
    S[threadIdx.x].tune = t;
    S[threadIdx.x].onepass = threadIdx.x == 0 ? onepass : 0;
  }
  if (threadIdx.x == 0) {
    *dst = v;
    base[0] = 0;
    base[1] = v.m;
  }
}

// Zero words (a launch costs a third of a small memset's call).
static __global__ void __launch_bounds__(256) k_zero(uint64_t *p, int64_t n) {
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x)
    p[i] = 0;
}

// True in every thread of the grid's last block to get here (the others'
// writes are then visible to it).  The ticket is left at zero.
__device__ __forceinline__ bool last_block(uint32_t *ticket) {
  __shared__ uint32_t s_last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    s_last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    if (s_last) {
      *ticket = 0;
      __threadfence();
    }
  }
  __syncthreads();
  return s_last != 0;
}

// Class offsets into the row list; resets the work counters.
__device__ __forceinline__ void sched_offsets(Sched *S) {
  int64_t o = 0;
  for (int c = 0; c < NCLS; ++c) {
    S->off[c] = o;
    S->cur[c] = o;
    S->next[c] = 0;
    o += *(volatile int64_t *)&S->cnt[c];
  }
  S->work = 0;
  S->work2 = 0;
  S->work3 = 0;
  S->rank_left = 0;
  S->rule = row_rule(*(volatile int64_t *)&S->total, *(volatile int64_t *)&S->nonempty);
}

// int32 row offsets widened to int64 (operands of mixed offset widths).
static __global__ void k_widen(const int32_t *src, int64_t n, int64_t *dst) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i < n) dst[i] = src[i];
}

// New operand arrays for a plan's numeric re-run; the sortedness found by the
// symbolic pass is kept.
template <typename PT, typename VT>
__global__ void k_set_operands(ProdDev<PT, VT> *dst, ProdDev<PT, VT> v) {
  const int32_t sorted = dst->b_sorted, strict = dst->b_strict;
  const void *ep = dst->Ep;  // the addend stays the symbolic call's
  const int32_t *ej = dst->Ej;
  const VT *ex = dst->Ex;
  const int32_t eb = dst->ep_bits;
  *dst = v;
  dst->b_sorted = sorted;
  dst->b_strict = strict;
  dst->Ep = ep;
  dst->Ej = ej;
  dst->Ex = ex;
  dst->ep_bits = eb;
}

template <typename PT, typename VT>
__global__ void k_set_out(ProdDev<PT, VT> *dst, int32_t *Cj, VT *Cx, void *Cp,
                          int cp_bits) {
  dst->Cj = Cj;
  dst->Cx = Cx;
  dst->Cp = Cp;
  dst->cp_bits = cp_bits;
}

// One warp per B row: set *flag = 0 if some row is not strictly increasing
// (the cursor sweep of the DENSE numeric class relies on sorted B rows).
template <typename PT>
__global__ void k_check_sorted_rows(const PT *Bp, const int32_t *Bj,
                                    int64_t nb, int32_t *flag) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = (int64_t(gridDim.x) * blockDim.x) >> 5;
  bool bad = false;
  for (int64_t r = warp; r < nb; r += nwarps) {
    const int64_t b0 = Bp[r], b1 = Bp[r + 1];
    for (int64_t q = b0 + lane; q + 1 < b1; q += 32)
      if (Bj[q] >= Bj[q + 1]) bad = true;
  }
  if (__any_sync(0xffffffffu, bad) && lane == 0) *flag = 0;
}

// Are all of B's rows strictly increasing?  One streaming pass: the places
// where a column is not above the one before it, less those between two rows,
// are none.  rec: a record of zero total and ticket, left so.
template <typename PT, typename VT>
__global__ void __launch_bounds__(256)
    k_check_strict(const PT *__restrict__ Bp, const int32_t *__restrict__ Bj, int64_t nb, Sched *rec,
                   ProdDev<PT, VT> *prod) {
  constexpr int U = 8;
  phase_begin();
  const int64_t stride = int64_t(gridDim.x) * blockDim.x;
  const int64_t t = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31;
  const int64_t first = int64_t(Bp[0]), end = int64_t(Bp[nb]);
  int64_t n = 0;
  for (int64_t q = first + t - lane; q + 1 < end; q += stride * U) {  // a warp's 32, uniform
    int32_t c[U], z[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t p = q + u * stride + lane;
      c[u] = p < end ? __ldg(Bj + p) : 0;
      z[u] = lane == 31 && p + 1 < end ? __ldg(Bj + p + 1) : 0;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int32_t up = __shfl_down_sync(0xffffffffu, c[u], 1);
      n += q + u * stride + lane + 1 < end && c[u] >= (lane < 31 ? up : z[u]);
    }
  }
  for (int64_t r = t; r < nb; r += stride) {
    const int64_t b0 = int64_t(__ldg(Bp + r)), b1 = int64_t(__ldg(Bp + r + 1));
    if (b1 > b0 && b1 < end) n -= __ldg(Bj + b1 - 1) >= __ldg(Bj + b1);
  }
  n = warp_sum(n);
  if ((threadIdx.x & 31) == 0 && n != 0) atomicAdd((unsigned long long *)&rec->total, (unsigned long long)n);
  if (last_block(&rec->ticket) && threadIdx.x == 0) {
    prod->b_strict = *(volatile int64_t *)&rec->total == 0;
    rec->total = 0;
  }
}

// ---------------------------------------------------------------------------
// Phase 0: mults per row and symbolic classes (one warp per row, shuffle
// reduction), block-aggregated class counts.
// Rows of at most this many A entries are walked by one lane in k_row_mults.
constexpr int kThreadRowMax = 64;
// ... and rows of more than this many are listed for k_row_mults_long (a CTA
// per row took 0.42 ms on the 119-entry rows of the Galerkin R·AP, a warp per
// row 0.1 ms).
constexpr int kLongRow = 256;
// A entries a one-pass candidate looks at for repeated columns.
constexpr int kHintEntries = 8;

// Products per row (rowf), the symbolic class counts, the product total, the
// sum of min(products, ncols) and the longest A row; with `finish` the last
// block turns the class counts into list offsets.  A warp takes 32 rows at
// a time: lane i walks row i's A entries itself (4 entries per step, so the
// loads of 32 rows are in flight together) when the row has at most
// kThreadRowMax entries, and the whole warp walks each longer row; class
// counts are aggregated per warp before the shared atomics (rows of one class
// would otherwise all hit one counter).  One warp per row, as first built,
// took 0.8 ms on the 2.1M rows of the Galerkin A·P (27 entries each): four
// dependent loads per row, one row per warp at a time.
//
// longs: the rows of more than kLongRow entries are listed there instead
// (k_row_mults_long): R-MAT's hub rows are neighbours, and the warp that held
// 32 of them was the pass (order 2^18, 16 draws a row: 0.58 ms).  Without a
// list the warp keeps 8 loads per lane in flight on such a row.
template <typename PT, typename VT>
__global__ void __launch_bounds__(256) k_row_mults(
    const ProdDev<PT, VT> *prods, const int64_t *base, int nprod, int64_t R,
    int64_t *rowf, Sched *S, int32_t *rowc = nullptr, int finish = 0, uint64_t *longs = nullptr) {
  __shared__ unsigned long long s_cnt[NCLS], s_cand[NCLS];
  __shared__ unsigned long long s_tot, s_up, s_ne;
  __shared__ long long s_maxa;
  if (threadIdx.x < NCLS) s_cnt[threadIdx.x] = s_cand[threadIdx.x] = 0;
  if (threadIdx.x == 0) s_tot = s_up = s_ne = 0, s_maxa = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int64_t warp = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = (int64_t(gridDim.x) * blockDim.x) >> 5;
  const int64_t ntiles = (R + 31) / 32;
  unsigned long long tot = 0, up = 0, ne = 0;
  long long maxa = 0;
  for (int64_t tile = warp; tile < ntiles; tile += nwarps) {
    const int64_t g = tile * 32 + lane;
    const bool valid = g < R;
    int p = 0;
    int64_t r = 0, a0 = 0, a1 = 0;
    const int32_t *Aj = nullptr;
    const PT *Bp = nullptr;
    if (valid) {
      p = find_prod(base, nprod, g);
      r = g - base[p];
      const PT *Ap = prods[p].Ap;
      Aj = prods[p].Aj;
      Bp = prods[p].Bp;
      a0 = int64_t(Ap[r]);
      a1 = int64_t(Ap[r + 1]);
    }
    const int64_t len = a1 - a0;
    const bool mine = len <= kThreadRowMax;  // rows past R have len 0
    const int tmax = int(__reduce_max_sync(0xffffffffu, mine ? unsigned(len) : 0u));
    int64_t f = 0;
    for (int t = 0; t < tmax; t += 4) {
      int64_t k[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) k[u] = mine && t + u < len ? int64_t(__ldg(Aj + a0 + t + u)) : -1;
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (k[u] >= 0) f += int64_t(__ldg(Bp + k[u] + 1)) - int64_t(__ldg(Bp + k[u]));
    }
    const bool listed = longs && len > kLongRow;
    if (const unsigned lm = __ballot_sync(0xffffffffu, listed)) {
      unsigned long long at = 0;
      if (lane == 0) at = atomicAdd(&S->nlong, (unsigned long long)__popc(lm));
      at = __shfl_sync(0xffffffffu, at, 0);
      if (listed) longs[at + __popc(lm & ((1u << lane) - 1u))] = (uint64_t(p) << 40) | uint64_t(r);
    }
    for (unsigned lr = __ballot_sync(0xffffffffu, !mine && !listed); lr; lr &= lr - 1) {
      const int j = __ffs(lr) - 1;
      const int pj = __shfl_sync(0xffffffffu, p, j);
      const int64_t b0 = __shfl_sync(0xffffffffu, a0, j), b1 = __shfl_sync(0xffffffffu, a1, j);
      const int32_t *Ajj = prods[pj].Aj;
      const PT *Bpj = prods[pj].Bp;
      int64_t sum = 0;
      for (int64_t q = b0; q < b1; q += 32 * 8) {
        int32_t k[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) k[u] = q + u * 32 + lane < b1 ? __ldg(Ajj + q + u * 32 + lane) : -1;
#pragma unroll
        for (int u = 0; u < 8; ++u)
          if (k[u] >= 0) sum += int64_t(__ldg(Bpj + k[u] + 1)) - int64_t(__ldg(Bpj + k[u]));
      }
      sum = warp_sum(sum);
      if (lane == j) f = sum;
    }
    // One-pass candidates too large for a warp's full table also need their
    // products to repeat columns: a row counts, over its first kHintEntries A
    // entries, those whose B row starts on the same column as the previous
    // entry's (0.5-0.6 of them on the Galerkin rows, 0.002 on uniform-random
    // rows); a few loads per such row.
    int same = 0, seen = 0;
    {
      const int64_t fe = f < (valid ? prods[p].n : 0) ? f : (valid ? prods[p].n : 0);
      const bool need = S->onepass && valid && !listed && fe > 0 && fe <= S->tune.sym[2] &&
                        int64_t(S->tune.load) * fe > 2 * kCappedCols;
      if (__any_sync(0xffffffffu, need)) {
        const int32_t *Bj = valid ? prods[p].Bj : nullptr;
        seen = need ? int(len < kHintEntries ? len : kHintEntries) : 0;
        int prev = -2;
        for (int t = 0; t < seen; ++t) {
          const int64_t k = __ldg(Aj + a0 + t);
          const int64_t q0 = int64_t(__ldg(Bp + k)), q1 = int64_t(__ldg(Bp + k + 1));
          const int first = q1 > q0 ? __ldg(Bj + q0) : -1;
          same += first >= 0 && first == prev;
          prev = first;
        }
      }
    }
    int c = -1, left = -1;
    if (valid && !listed) {
      if (prods[p].Ej) {  // the addend's entries count as products of the row
        int64_t e0, e1;
        addend_row(prods[p], r, e0, e1);
        f += e1 - e0;
      }
      rowf[g] = f;
      const int64_t n = prods[p].n;
      c = sym_class(f, n, S->tune);
      // one-pass rows: their scratch bound; the class they leave is kept
      // (cand) in case the product takes the two-pass path after all
      // candidates: rows whose bound fits a warp's full table, and larger
      // ones whose products look like repeating columns (their 64-slot
      // attempt is likely to hold the row)
      const bool one = S->onepass && onepass_row(f, n, S->tune) &&
                       (onepass_full(f, n, S->tune) || (seen > 1 && 4 * same >= seen - 1));
      if (one) {
        left = c;
        c = CLS_ONEPASS;
      }
      // zero, or a one-pass row's scratch bound, until the symbolic kernels
      // write the counts of the rows that have products
      if (rowc) rowc[g] = one ? int32_t(onepass_bound(f, n, S->tune)) : 0;
      if (c >= 0) ne += 1;
      tot += f;
      up += f < n ? f : n;
      if (len > maxa) maxa = len;
    }
    // one shared atomic per class present in the warp
    for (unsigned todo = __ballot_sync(0xffffffffu, c >= 0); todo;) {
      const int cl = __shfl_sync(0xffffffffu, c, __ffs(todo) - 1);
      const unsigned m = __ballot_sync(0xffffffffu, c == cl);
      if (lane == __ffs(m) - 1) atomicAdd(&s_cnt[cl], (unsigned long long)__popc(m));
      todo &= ~m;
    }
    for (unsigned todo = __ballot_sync(0xffffffffu, left >= 0); todo;) {
      const int cl = __shfl_sync(0xffffffffu, left, __ffs(todo) - 1);
      const unsigned m = __ballot_sync(0xffffffffu, left == cl);
      if (lane == __ffs(m) - 1) atomicAdd(&s_cand[cl], (unsigned long long)__popc(m));
      todo &= ~m;
    }
  }
  tot = warp_sum(tot);
  up = warp_sum(up);
  ne = warp_sum(ne);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const long long other = __shfl_xor_sync(0xffffffffu, maxa, o);
    maxa = other > maxa ? other : maxa;
  }
  if (lane == 0) {
    atomicAdd(&s_tot, tot);
    atomicAdd(&s_up, up);
    atomicAdd(&s_ne, ne);
    atomicMax(&s_maxa, maxa);
  }
  __syncthreads();
  if (threadIdx.x < NCLS && s_cnt[threadIdx.x])
    atomicAdd((unsigned long long *)&S->cnt[threadIdx.x], s_cnt[threadIdx.x]);
  if (threadIdx.x < NCLS && s_cand[threadIdx.x])
    atomicAdd((unsigned long long *)&S->cand[threadIdx.x], s_cand[threadIdx.x]);
  if (threadIdx.x == 0) {
    atomicAdd((unsigned long long *)&S->total, s_tot);
    atomicAdd((unsigned long long *)&S->upper, s_up);
    atomicAdd((unsigned long long *)&S->nonempty, s_ne);
    atomicMax((long long *)&S->max_a_row, s_maxa);
  }
  if (finish && last_block(&S->ticket) && threadIdx.x == 0) sched_offsets(S);
}

// The rows k_row_mults listed (more than kLongRow A entries), a CTA each,
// with the same results per row.
template <typename PT, typename VT>
__global__ void __launch_bounds__(256) k_row_mults_long(
    const ProdDev<PT, VT> *prods, const int64_t *base, int64_t *rowf, Sched *S, int32_t *rowc,
    const uint64_t *longs) {
  __shared__ int64_t part[8];
  __shared__ unsigned long long s_cnt[NCLS], s_cand[NCLS];
  const int tid = threadIdx.x, lane = tid & 31;
  if (tid < NCLS) s_cnt[tid] = s_cand[tid] = 0;
  const int64_t n = int64_t(S->nlong);
  unsigned long long tot = 0, up = 0, ne = 0;  // thread 0's
  long long maxa = 0;
  for (int64_t i = blockIdx.x; i < n; i += gridDim.x) {
    const int p = int(longs[i] >> 40);
    const int64_t r = int64_t(longs[i] & ((uint64_t(1) << 40) - 1));
    const ProdDev<PT, VT> &P = prods[p];
    const int32_t *__restrict__ Aj = P.Aj;
    const PT *__restrict__ Bp = P.Bp;
    const int64_t a0 = int64_t(P.Ap[r]), a1 = int64_t(P.Ap[r + 1]);
    int64_t sum = 0;
    for (int64_t q = a0 + tid; q < a1; q += 256 * 4) {
      int32_t k[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) k[u] = q + u * 256 < a1 ? __ldg(Aj + q + u * 256) : -1;
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (k[u] >= 0) sum += int64_t(__ldg(Bp + k[u] + 1)) - int64_t(__ldg(Bp + k[u]));
    }
    sum = warp_sum(sum);
    if (lane == 0) part[tid >> 5] = sum;
    __syncthreads();
    if (tid == 0) {
      int64_t f = 0;
      for (int w = 0; w < 8; ++w) f += part[w];
      const int64_t g = base[p] + r;
      bool repeats = false;  // as in k_row_mults: kHintEntries (< kLongRow) entries
      if (S->onepass && onepass_row(f, P.n, S->tune) && !onepass_full(f, P.n, S->tune)) {
        int same = 0, prev = -2;
        for (int t = 0; t < kHintEntries; ++t) {
          const int64_t k = __ldg(Aj + a0 + t);
          const int64_t q0 = int64_t(__ldg(Bp + k)), q1 = int64_t(__ldg(Bp + k + 1));
          const int first = q1 > q0 ? __ldg(P.Bj + q0) : -1;
          same += first >= 0 && first == prev;
          prev = first;
        }
        repeats = 4 * same >= kHintEntries - 1;
      }
      if (P.Ej) {
        int64_t e0, e1;
        addend_row(P, r, e0, e1);
        f += e1 - e0;
      }
      rowf[g] = f;
      int c = sym_class(f, P.n, S->tune);
      const bool one = S->onepass && onepass_row(f, P.n, S->tune) &&
                       (onepass_full(f, P.n, S->tune) || repeats);
      if (one) {
        ++s_cand[c];
        c = CLS_ONEPASS;
      }
      if (rowc) rowc[g] = one ? int32_t(onepass_bound(f, P.n, S->tune)) : 0;
      if (c >= 0) {
        ++s_cnt[c];
        ++ne;
      }
      tot += (unsigned long long)f;
      up += (unsigned long long)(f < P.n ? f : P.n);
      if (a1 - a0 > maxa) maxa = a1 - a0;
    }
    __syncthreads();
  }
  if (tid == 0 && maxa > 0) {
    for (int c = 0; c < NCLS; ++c) {
      if (s_cnt[c]) atomicAdd((unsigned long long *)&S->cnt[c], s_cnt[c]);
      if (s_cand[c]) atomicAdd((unsigned long long *)&S->cand[c], s_cand[c]);
    }
    atomicAdd((unsigned long long *)&S->total, tot);
    atomicAdd((unsigned long long *)&S->upper, up);
    atomicAdd((unsigned long long *)&S->nonempty, ne);
    atomicMax((long long *)&S->max_a_row, maxa);
  }
}

// The count pass of R rows: rowf, the record's class counts and sums.  longs
// (R entries): the list of long rows of products of kFuseRows rows or more,
// whose count takes a launch of its own.
template <typename PT, typename VT>
static inline void launch_row_mults(tspg_ctx *ctx, cudaStream_t s, const ProdDev<PT, VT> *prods,
                                    const int64_t *base, int nprod, int64_t R, int64_t *rowf,
                                    Sched *S, int32_t *rowc, int finish, uint64_t *longs) {
  const unsigned g = unsigned((R * 32 + 255) / 256 < int64_t(ctx->num_sms) * 16
                                  ? (R * 32 + 255) / 256 : int64_t(ctx->num_sms) * 16);
  k_row_mults<PT, VT><<<g, 256, 0, s>>>(prods, base, nprod, R, rowf, S, rowc, finish, longs);
  ctx->launches += 1;
  if (longs) {
    k_row_mults_long<PT, VT><<<ctx->num_sms * 8, 256, 0, s>>>(prods, base, rowf, S, rowc, longs);
    ctx->launches += 1;
  }
}

// The one-pass rows of a symbolic record go back to the classes they left
// (the product takes the two-pass path after all).
static __global__ void k_fold_onepass(Sched *S) {
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    for (int c = 0; c < NCLS; ++c) S->cnt[c] += S->cand[c];
    S->cnt[CLS_ONEPASS] = 0;
    S->onepass = 0;
  }
}

// The record of the one-pass rows sent back to the two-pass path (their
// list: the deferred rows), counted as 256-thread symbolic rows.
static __global__ void k_defer_setup(const Sched *S, Sched *D) {
  if (threadIdx.x == 0 && blockIdx.x == 0) D->cnt[CLS_G256] = int64_t(S->ndefer);
}

static __global__ void k_sched_offsets(Sched *S) {
  if (threadIdx.x == 0 && blockIdx.x == 0) sched_offsets(S);
}

// The output arrays of a single product (set: they go into its descriptor).
struct OutArgs {
  int32_t *Cj = nullptr;
  void *Cx = nullptr;
  void *Cp = nullptr;
  int32_t cp_bits = 0;
  int16_t set = 0;
  int16_t finish = 0;
};

// Scatter rows into the class lists.  mode 0: symbolic (class from rowf);
// mode 1: numeric (class from rowc) which also writes the output row offsets
// of each product, and whose last block (out.finish) makes the record ready
// for the numeric kernels and for another numeric run of a plan.
template <typename PT, typename VT, int MODE>
__global__ void __launch_bounds__(256) k_scatter(
    ProdDev<PT, VT> *prods, const int64_t *base, int nprod, int64_t R,
    const int64_t *rowf, const int32_t *rowc, const int64_t *cp, Sched *S,
    uint64_t *list, OutArgs out = OutArgs()) {
  __shared__ unsigned long long s_cnt[NCLS], s_base[NCLS];
  if (threadIdx.x < NCLS) s_cnt[threadIdx.x] = 0;
  __syncthreads();
  const int64_t g = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  int c = -1, p = 0;
  int64_t r = 0;
  unsigned long long my = 0;
  if (g < R) {
    p = find_prod(base, nprod, g);
    r = g - base[p];
    if (MODE == 0) {
      c = sym_class(rowf[g], prods[p].n, S->tune);
      if (S->onepass && rowc[g] > 0) c = CLS_ONEPASS;  // the count pass's choice (bound > 0)
    } else {
      c = num_class(rowc[g], rowf[g], S->tune, S[-1].rule);
      const int64_t off = cp[g] - cp[base[p]];
      void *const Cp = out.set ? out.Cp : prods[p].Cp;
      const bool narrow = (out.set ? out.cp_bits : prods[p].cp_bits) == 32;
      if (narrow) ((int32_t *)Cp)[r] = (int32_t)off;
      else ((int64_t *)Cp)[r] = off;
      if (r == prods[p].m - 1) {
        const int64_t end = cp[g + 1] - cp[base[p]];
        if (narrow) ((int32_t *)Cp)[r + 1] = (int32_t)end;
        else ((int64_t *)Cp)[r + 1] = end;
      }
    }
  }
  if (MODE == 1 && out.set && blockIdx.x == 0 && threadIdx.x == 0) {
    prods[0].Cj = out.Cj;
    prods[0].Cx = (VT *)out.Cx;
    prods[0].Cp = out.Cp;
    prods[0].cp_bits = out.cp_bits;
  }
  // each class present in the warp takes its slots with one shared atomic
  const int lane = threadIdx.x & 31;
  for (unsigned todo = __ballot_sync(0xffffffffu, c >= 0); todo;) {
    const int leader = __ffs(todo) - 1;
    const int cl = __shfl_sync(0xffffffffu, c, leader);
    const unsigned m = __ballot_sync(0xffffffffu, c == cl);
    unsigned long long b = 0;
    if (lane == leader) b = atomicAdd(&s_cnt[cl], (unsigned long long)__popc(m));
    b = __shfl_sync(0xffffffffu, b, leader);
    if (c == cl) my = b + __popc(m & ((1u << lane) - 1u));
    todo &= ~m;
  }
  __syncthreads();
  if (threadIdx.x < NCLS) {
    s_base[threadIdx.x] =
        s_cnt[threadIdx.x]
            ? atomicAdd((unsigned long long *)&S->cur[threadIdx.x],
                        s_cnt[threadIdx.x])
            : 0;
  }
  __syncthreads();
  if (c >= 0) list[s_base[c] + my] = (uint64_t(p) << 40) | uint64_t(r);
  phase_end();
  if (MODE == 1 && out.finish && last_block(&S->ticket) && threadIdx.x == 0) sched_offsets(S);
}

// Products whose A has zero rows still need rowptr[0] = 0.
template <typename PT, typename VT>
__global__ void k_zero_rowptr(ProdDev<PT, VT> *prods, int nprod) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p < nprod && prods[p].m == 0) {
    if (prods[p].cp_bits == 32) ((int32_t *)prods[p].Cp)[0] = 0;
    else ((int64_t *)prods[p].Cp)[0] = 0;
  }
}

// ---------------------------------------------------------------------------
// Device-wide exclusive scan of int32 row counts into int64 offsets
// (reduce, scan of partials, final).  cp has R + 1 entries.
constexpr int kScanThreads = 512;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;

static __global__ void __launch_bounds__(kScanThreads)
    k_scan_reduce(const int32_t *in, int64_t R, int64_t *partial, uint32_t *ticket = nullptr) {
  __shared__ int64_t tmp[kScanThreads / 32 + 1];
  const int64_t t0 = int64_t(blockIdx.x) * kScanTile;
  int64_t s = 0;
  for (int i = 0; i < kScanItems; ++i) {
    const int64_t j = t0 + int64_t(i) * kScanThreads + threadIdx.x;
    if (j < R) s += in[j];
  }
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0) tmp[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    int64_t v = threadIdx.x < kScanThreads / 32 ? tmp[threadIdx.x] : 0;
    v = warp_sum(v);
    if (threadIdx.x == 0) partial[blockIdx.x] = v;
  }
  // the last block scans the partials in place (partial[nb] = total)
  if (ticket && last_block(ticket)) {
    const int64_t nb = gridDim.x;
    int64_t carry = 0;
    for (int64_t b0 = 0; b0 < nb; b0 += kScanThreads) {
      const int64_t j = b0 + threadIdx.x;
      const int64_t v = j < nb ? *(volatile int64_t *)(partial + j) : 0;
      int64_t tot;
      const int64_t ex = group_excl_scan<kScanThreads, int64_t>(v, tmp, 0, &tot);
      if (j < nb) partial[j] = carry + ex;
      carry += tot;
    }
    if (threadIdx.x == 0) partial[nb] = carry;
  }
}

// Single block: exclusive scan of nb partials in place; partial[nb] = total.
static __global__ void __launch_bounds__(1024) k_scan_partials(int64_t *partial,
                                                        int64_t nb) {
  __shared__ int64_t tmp[33];
  __shared__ int64_t carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (int64_t b0 = 0; b0 < nb; b0 += 1024) {
    const int64_t j = b0 + threadIdx.x;
    const int64_t v = j < nb ? partial[j] : 0;
    int64_t tot;
    const int64_t ex = group_excl_scan<1024, int64_t>(v, tmp, 0, &tot);
    if (j < nb) partial[j] = carry + ex;
    __syncthreads();
    if (threadIdx.x == 0) carry += tot;
    __syncthreads();
  }
  if (threadIdx.x == 0) partial[nb] = carry;
}

// What the symbolic phase of a single product leaves for the host, written
// from the device into mapped pinned memory (a stream sync then suffices; a
// device->host copy took 2.6 us each): nnz(C), the record's sums, the error
// word and the numeric class counts.
enum { HW_TOTAL = 0, HW_MULTS, HW_MAX_A, HW_ERR, HW_CNT };
struct HostWords {
  int64_t *words = nullptr;      // null: nothing is left
  const Sched *sym = nullptr;    // the symbolic record
  const int64_t *err = nullptr;  // the device error word
};

// One thread: the numeric record's list offsets and the host's words.
__device__ __forceinline__ void finish_symbolic(Sched *Snum, int64_t total, const HostWords &host) {
  sched_offsets(Snum);
  volatile int64_t *w = host.words;
  w[HW_TOTAL] = total;
  w[HW_MULTS] = host.sym->total;
  w[HW_MAX_A] = host.sym->max_a_row;
  w[HW_ERR] = *host.err;
  for (int c = 0; c < NCLS; ++c) w[HW_CNT + c] = *(volatile int64_t *)&Snum->cnt[c];
  __threadfence_system();
}

static __global__ void k_finish_symbolic(Sched *Snum, const int64_t *total, HostWords host) {
  if (threadIdx.x == 0) finish_symbolic(Snum, *total, host);
}

// Final pass of the scan; partial == null: the one block has everything.
// Also counts the numeric classes of the rows into *Snum (rowf given); with
// host.words the last block finishes the symbolic phase.
static __global__ void __launch_bounds__(kScanThreads)
    k_scan_final(const int32_t *in, int64_t R, const int64_t *partial,
                 int64_t nb, int64_t *out, Sched *Snum, const int64_t *rowf,
                 HostWords host = HostWords(), int64_t *host_total = nullptr) {
  __shared__ int64_t tmp[kScanThreads / 32 + 1];
  __shared__ unsigned long long s_cnt[NCLS];
  if (threadIdx.x < NCLS) s_cnt[threadIdx.x] = 0;
  __syncthreads();
  const int64_t t0 = int64_t(blockIdx.x) * kScanTile;
  // each thread owns kScanItems consecutive elements
  const int64_t j0 = t0 + int64_t(threadIdx.x) * kScanItems;
  int64_t v[kScanItems];
  int64_t s = 0;
  uint32_t packed = 0;  // 4-bit count per class (kScanItems <= 15)
  static_assert(kScanItems <= 15 && NCLS * 4 <= 32, "packed class counts");
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) {
    v[i] = (j0 + i < R) ? in[j0 + i] : 0;
    s += v[i];
    if (rowf && v[i] > 0) {
      const int c = num_class(v[i], rowf[j0 + i], Snum->tune, Snum[-1].rule);
      if (c >= 0) packed += 1u << (4 * c);
    }
  }
  // class counts: a warp reduction per class, one shared atomic per warp
  // (rows of one class would otherwise all hit one counter)
  if (rowf) {
#pragma unroll
    for (int c = 0; c < NCLS; ++c) {
      const unsigned x = __reduce_add_sync(0xffffffffu, (packed >> (4 * c)) & 15u);
      if ((threadIdx.x & 31) == 0 && x) atomicAdd(&s_cnt[c], (unsigned long long)x);
    }
  }
  int64_t tot;
  int64_t ex = group_excl_scan<kScanThreads, int64_t>(s, tmp, 0, &tot);
  if (partial) ex += partial[blockIdx.x];
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) {
    if (j0 + i < R) out[j0 + i] = ex;
    ex += v[i];
  }
  const int64_t total = partial ? partial[nb] : tot;
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) {
    out[R] = total;
    if (host_total) {
      *(volatile int64_t *)host_total = total;
      __threadfence_system();
    }
  }
  __syncthreads();
  if (threadIdx.x < NCLS && s_cnt[threadIdx.x])
    atomicAdd((unsigned long long *)&Snum->cnt[threadIdx.x], s_cnt[threadIdx.x]);
  if (host.words && last_block(&Snum->ticket) && threadIdx.x == 0)
    finish_symbolic(Snum, total, host);
}

// Row offsets of an output written in equal tiles of TILE source entries, whose
// CTAs write the offsets of the rows that start in them — unless some tile
// holds more than kTileRows rows (long runs of empty ones: a CTA would walk
// them alone; 1M rows of 600 entries: 15 ms a merge).  Then the tiles leave
// every source entry's output slot, counted from the tile's first, in pos, and
// this grid-wide pass takes each row's from there.  off: the tiles' first
// slots, off[ntiles] the total; a row starts at source entry Ap[r] (+ Bp[r]).
constexpr int64_t kTileRows = 4096;
template <int TILE, typename PTA, typename PTB>
__global__ void __launch_bounds__(256)
    k_tile_offsets(const PTA *__restrict__ Ap, const PTB *__restrict__ Bp, int64_t m,
                   const int64_t *__restrict__ off, int64_t ntiles,
                   const uint16_t *__restrict__ pos, void *Cp, int cp_bits) {
  const int64_t r = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (r > m) return;
  auto start = [&](int64_t q) {
    int64_t d = int64_t(__ldg(Ap + q)) - int64_t(__ldg(Ap));
    if (Bp) d += int64_t(__ldg(Bp + q)) - int64_t(__ldg(Bp));
    return d;
  };
  const int64_t d = start(r);
  const int64_t at = d < start(m) ? off[d / TILE] + pos[d] : off[ntiles];
  if (cp_bits == 32) ((int32_t *)Cp)[r] = int32_t(at);
  else ((int64_t *)Cp)[r] = at;
}

// Rows from which a step's last block no longer does what a small launch of
// its own can: every block then pays a fence and a ticket (2.1M rows: count
// pass +14 us, final scan +6 us, against 2-3 us a launch).
constexpr int64_t kFuseRows = 1 << 16;

// Exclusive scan of in[0, R) into out[0, R] (R > 0): one launch up to
// kScanTile rows, two below kFuseRows, else three.  S: a zeroed record (its
// ticket is used).
static inline void launch_scan(tspg_ctx *ctx, cudaStream_t s, const int32_t *in, int64_t R,
                               int64_t *partial, int64_t *out, Sched *S, const int64_t *rowf,
                               HostWords host = HostWords(), int64_t *host_total = nullptr) {
  const int64_t nb = (R + kScanTile - 1) / kScanTile;
  const bool fuse = R < kFuseRows;
  if (nb > 1) {
    k_scan_reduce<<<(unsigned)nb, kScanThreads, 0, s>>>(in, R, partial, fuse ? &S->ticket : nullptr);
    if (!fuse) k_scan_partials<<<1, 1024, 0, s>>>(partial, nb);
    ctx->launches += fuse ? 1 : 2;
  }
  k_scan_final<<<(unsigned)nb, kScanThreads, 0, s>>>(in, R, nb > 1 ? partial : nullptr, nb, out, S,
                                                     rowf, fuse ? host : HostWords(), host_total);
  ctx->launches += 1;
  if (host.words && !fuse) {
    k_finish_symbolic<<<1, 32, 0, s>>>(S, out + R, host);
    ctx->launches += 1;
  }
}

}  // namespace tspg
