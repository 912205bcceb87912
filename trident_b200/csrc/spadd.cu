// spadd.cu — merge of partial C tiles, C = A + B with the union pattern.
//
// Replaces cusparse_spgeam (include/cusparse_helpers.cuh:799-905: csrgeam2
// bufferSize + Nnz + compute, five stream syncs, the nnz through the host) and
// LocalMatrix::spadd (include/KokkosWrap.hpp:394-439: KK spadd symbolic +
// numeric).  Rows are sorted and duplicate-free, so both operands are sequences
// sorted by (row, column) and the union is one merge of the two.  It is cut
// into tiles of kMergeTile merged entries, whatever the rows' lengths: one
// thread per cut finds its row in the sum of the row offsets, then its place
// inside the row (merge path); a CTA merges a tile, each thread 7 entries,
// first counting, then writing.
//
// What bounds it: the serial merges and the two searches before them (about 30
// warp instructions per 32 entries and pass); the operands cross memory twice.
// R-MAT of order 2^18, 64 draws a row, A + B: 0.83 -> 0.43 ms against one warp
// per row merging 32-column chunks ranked by shuffles (about 400 instructions
// per 32 entries, hub rows in a kernel of their own); 0.49 ms with a tile's
// loads in loops of unknown length instead of all in flight.  Long runs of empty
// rows: 1M rows holding 300 + 300 entries 0.10 ms (a thread stepping over them
// row by row, and a CTA writing their offsets: 15 ms; a warp per row: 0.21 ms).
#include "internal.cuh"
#include "spgemm_kernels.cuh"

namespace tspg {

constexpr int kMergeThreads = 256;
constexpr int kMergePer = 7;  // merged entries per thread: odd, so that threads stepping through
                               // shared memory in step hit different banks
constexpr int kMergeTile = kMergeThreads * kMergePer;
// Row ends kept in shared memory.  A tile over more rows (runs of empty ones:
// it holds kMergeTile entries at most) searches the offsets for each entry's row.
constexpr int kMergeRows = 1024;

// A cut of the merged sequence before entry d: the row whose entries it falls
// into (the last one starting at or before d), the first row starting at or
// after d, and the entries of A and B (from their first) before it.
struct MergeCut {
  int64_t row, first, i, j;
};

template <typename PTA, typename PTB>
__global__ void __launch_bounds__(128)
    k_merge_cuts(int64_t m, const PTA *__restrict__ Ap, const int32_t *__restrict__ Aj,
                 const PTB *__restrict__ Bp, const int32_t *__restrict__ Bj, int64_t ntiles,
                 MergeCut *cuts, Sched *rec) {
  const int64_t t = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (t == 0) rec->ticket = 0;  // of the scan to come
  if (t > ntiles) return;
  const int64_t ab = int64_t(Ap[0]), bb = int64_t(Bp[0]);
  auto start = [&](int64_t r) { return int64_t(__ldg(Ap + r)) - ab + int64_t(__ldg(Bp + r)) - bb; };
  const int64_t total = start(m);
  const int64_t d = t * kMergeTile < total ? t * kMergeTile : total;
  int64_t lo = 0, hi = m;  // the last row in [0, m] with start <= d
  while (lo < hi) {
    const int64_t mid = (lo + hi + 1) >> 1;
    if (start(mid) <= d) lo = mid; else hi = mid - 1;
  }
  MergeCut c;
  c.row = lo;
  if (start(lo) < d) {
    c.first = lo + 1;
  } else {
    int64_t a = 0, z = lo;  // the first row with start >= d
    while (a < z) {
      const int64_t mid = (a + z) >> 1;
      if (start(mid) < d) a = mid + 1; else z = mid;
    }
    c.first = a;
  }
  c.i = int64_t(__ldg(Ap + lo)) - ab;
  c.j = int64_t(__ldg(Bp + lo)) - bb;
  if (lo < m) {
    // A before B on equal columns: among the row's first q merged entries are
    // x of A, the least x with A[x] > B[q - 1 - x]
    const int64_t la = int64_t(__ldg(Ap + lo + 1)) - ab - c.i, lb = int64_t(__ldg(Bp + lo + 1)) - bb - c.j;
    const int64_t q = d - c.i - c.j;
    const int32_t *aj = Aj + ab + c.i, *bj = Bj + bb + c.j;
    int64_t x = q > lb ? q - lb : 0, y = q < la ? q : la;
    while (x < y) {
      const int64_t mid = (x + y) >> 1;
      if (__ldg(aj + mid) <= __ldg(bj + q - 1 - mid)) x = mid + 1; else y = mid;
    }
    c.i += x;
    c.j += q - x;
  }
  cuts[t] = c;
}

// One tile: WRITE = false leaves its number of output entries in tilec[tile]
// and checks the order of the rows; WRITE = true writes them from off[tile] on,
// and the offsets of the rows that start in the tile (pos given: their entries'
// slots, for k_tile_offsets; order[2] = 1 asks for that).  A column in both rows leaves with A's entry (the two
// values added); B's entry of the pair is a "dup" and leaves nothing, so entry
// x of the tile goes to slot x - (dups before x).
//
// The order check (order[0] = 1: a row descends, order[1] = 1: a row holds a
// column twice): a cut inside a row that is not sorted may lie before the cut
// it follows, so a tile with a negative share of A or B is left alone.  With
// both shares at or above 0 every index stays inside the tile, whatever the
// columns: the cursors start inside their row and move by one entry a step.
// Each entry is compared with the one before it in its row by the thread that
// merges it; that no entry is passed over is checked by comparing every
// thread's end with the next one's start (in sorted rows they agree).
template <bool WRITE, typename PTA, typename PTB, typename VT>
__global__ void __launch_bounds__(kMergeThreads)
    k_merge_tiles(int64_t m, const PTA *__restrict__ Ap, const int32_t *__restrict__ Aj,
                  const VT *__restrict__ Ax, const PTB *__restrict__ Bp,
                  const int32_t *__restrict__ Bj, const VT *__restrict__ Bx, int64_t ntiles,
                  const MergeCut *__restrict__ cuts, int32_t *tilec, volatile int64_t *order,
                  const int64_t *off, uint16_t *pos, void *Cp, int cp_bits, int32_t *Cj, VT *Cx) {
  __shared__ VT sv[WRITE ? kMergeTile + 2 : 1];       // A's values, then B's, one more of B
  __shared__ int32_t sc[kMergeTile + 2];              // one column of A before, A's, B's, one of B
  __shared__ uint32_t send[kMergeRows];               // row ends in the tile
  __shared__ uint32_t sfrom[kMergeTile];              // ends of the row that starts at an entry, so that
                                                      // nobody steps over empty rows
  __shared__ uint16_t sdup[kMergeThreads + 1];        // dups before a thread's entries; counting: A's before them
  __shared__ uint8_t sbit[kMergeThreads + 1];         // a thread's dups, bit per entry
  __shared__ int wsum[kMergeThreads / 32];
  __shared__ int32_t sb0;  // one column of B before
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int64_t ab = int64_t(Ap[0]), bb = int64_t(Bp[0]);
  const MergeCut c0 = cuts[blockIdx.x], c1 = cuts[blockIdx.x + 1];
  const int nA = int(c1.i - c0.i), nB = int(c1.j - c0.j), n = nA + nB;
  if (!WRITE && (nA < 0 || nB < 0)) {  // uniform
    if (tid == 0) {
      tilec[blockIdx.x] = 0;
      order[0] = 1;
    }
    return;
  }
  const int32_t *__restrict__ aj = Aj + ab + c0.i;
  const int32_t *__restrict__ bj = Bj + bb + c0.j;
  const int64_t rl = c1.row < m ? c1.row : m - 1;  // the last row with entries here, or one after
  const int64_t R = rl - c0.row + 1;
  const bool small = R <= kMergeRows;
  int32_t *sa = sc + 1, *sb = sc + 1 + nA;
  {  // all of a thread's loads in flight
    const VT *__restrict__ ax = Ax + ab + c0.i, *__restrict__ bx = Bx + bb + c0.j;
    int32_t lc[kMergePer];
    VT lv[kMergePer];
#pragma unroll
    for (int t = 0; t < kMergePer; ++t) {
      const int x = tid + t * kMergeThreads;
      if (x < n) {
        lc[t] = x < nA ? __ldg(aj + x) : __ldg(bj + (x - nA));
        if (WRITE) lv[t] = x < nA ? __ldg(ax + x) : __ldg(bx + (x - nA));
      }
    }
#pragma unroll
    for (int t = 0; t < kMergePer; ++t) {
      const int x = tid + t * kMergeThreads;
      if (x < n) {
        sa[x] = lc[t];
        if (WRITE) sv[x] = lv[t];
      }
    }
  }
  if (tid == 0) {
    // the pair cut by the tile's edge: A's entry before the tile (same row as
    // its first), B's entry after it (same row as its last)
    const int64_t a0 = int64_t(Ap[c0.row]) - ab;
    sc[0] = c0.row < m && c0.i > a0 ? __ldg(aj - 1) : -1;
    if (!WRITE) {
      const int64_t b0 = int64_t(Bp[c0.row]) - bb;
      sb0 = c0.row < m && c0.j > b0 ? __ldg(bj - 1) : -1;
    }
    int32_t after = -1;
    if (c1.row < m && int64_t(Ap[c1.row]) - ab + int64_t(Bp[c1.row]) - bb < c1.i + c1.j &&
        c1.j < int64_t(Bp[c1.row + 1]) - bb) {
      after = __ldg(bj + nB);
      if (WRITE) sv[n] = __ldg(Bx + bb + c0.j + nB);
    }
    sb[nB] = after;
  }
  // ends of row c0.row + k, clipped to the tile: A's, B's << 16
  auto row_end = [&](int64_t k) {
    const int64_t a = int64_t(__ldg(Ap + c0.row + k + 1)) - ab - c0.i;
    const int64_t b = int64_t(__ldg(Bp + c0.row + k + 1)) - bb - c0.j;
    return uint32_t(a < nA ? a : nA) | uint32_t(b < nB ? b : nB) << 16;
  };
  auto both = [](uint32_t e) { return int((e & 0xffffu) + (e >> 16)); };
  if (small) {
    for (int k0 = w * 32; k0 < int(R); k0 += kMergeThreads) {
      const int k = k0 + lane;
      const uint32_t e = k < int(R) ? row_end(k) : 0u, b = lane == 0 && k > 0 ? row_end(k - 1) : 0u;
      const uint32_t up = __shfl_up_sync(0xffffffffu, e, 1);
      const int s = both(lane > 0 ? up : b);
      if (k < int(R)) {
        send[k] = e;
        if (both(e) > s) sfrom[s] = e;
      }
    }
  } else {  // far more rows than entries: the row of every entry, by a search
    for (int x = tid; x < n; x += kMergeThreads) {
      const int64_t d = c0.i + c0.j + x + ab + bb;
      int64_t lo = c0.row, hi = rl;
      while (lo < hi) {
        const int64_t mid = (lo + hi) >> 1;
        if (int64_t(__ldg(Ap + mid + 1)) + int64_t(__ldg(Bp + mid + 1)) > d) hi = mid; else lo = mid + 1;
      }
      sfrom[x] = row_end(lo - c0.row);
    }
  }
  __syncthreads();
  auto ends = [&](int64_t k) { return small ? send[k] : row_end(k); };
  const int x0 = tid * kMergePer;
  int32_t col[kMergePer];
  VT val[kMergePer];
  unsigned dups = 0;
  int i = nA;
  bool down = false, twice = false;
  if (!WRITE && x0 >= n) sdup[tid] = uint16_t(nA);
  if (x0 < n) {
    int64_t lo = 0, hi = R - 1;  // the first row that ends past x0
    while (lo < hi) {
      const int64_t mid = (lo + hi) >> 1;
      if (both(ends(mid)) > x0) hi = mid; else lo = mid + 1;
    }
    const int64_t k = lo;
    const uint32_t ks = k > 0 ? ends(k - 1) : 0u, ke = ends(k);
    const int as = int(ks & 0xffffu), bs = int(ks >> 16);
    int ae = int(ke & 0xffffu), be = int(ke >> 16);
    // the row's merge path at x0
    const int q = x0 - as - bs, la = ae - as, lb = be - bs;
    int x = q > lb ? q - lb : 0, y = q < la ? q : la;
    while (x < y) {
      const int mid = (x + y) >> 1;
      if (sa[as + mid] <= sb[bs + q - 1 - mid]) x = mid + 1; else y = mid;
    }
    i = as + x;
    int j = bs + q - x;
    if (!WRITE) sdup[tid] = uint16_t(i);
    // columns at the cursors (INT32_MAX past the row's end) and of the A entry
    // before i (-1 when that is not in this row)
    int32_t ca = i < ae ? sa[i] : INT32_MAX, cb = j < be ? sb[j] : INT32_MAX;
    int32_t pa = i > as ? sa[i - 1] : k == 0 && i == 0 ? sc[0] : -1;
    int32_t pb = WRITE ? -1 : j > bs ? sb[j - 1] : k == 0 && j == 0 ? sb0 : -1;
#pragma unroll
    for (int t = 0; t < kMergePer; ++t) {
      if (x0 + t < n) {
        if (i == ae && j == be) {  // the next row with entries
          const uint32_t e = sfrom[x0 + t];
          ae = int(e & 0xffffu);
          be = int(e >> 16);
          ca = i < ae ? sa[i] : INT32_MAX;
          cb = j < be ? sb[j] : INT32_MAX;
          pa = pb = -1;
        }
        if (ca <= cb) {  // (an exhausted A row has ca = INT32_MAX > any column)
          col[t] = ca;
          if (WRITE) {
            // B's entry of the pair, possibly the one after the tile
            const bool pair = cb == ca || (j == nB && i == nA - 1 && sb[nB] == ca);
            val[t] = sv[i];
            if (pair) val[t] += sv[nA + j];
          } else {
            down |= pa > ca;
            twice |= pa == ca;
          }
          pa = ca;
          ++i;
          ca = i < ae ? sa[i] : INT32_MAX;
        } else {
          col[t] = cb;
          if (cb == pa) dups |= 1u << t;
          if (WRITE) {
            val[t] = sv[nA + j];
          } else {
            down |= pb > cb;
            twice |= pb == cb;
            pb = cb;
          }
          ++j;
          cb = j < be ? sb[j] : INT32_MAX;
        }
      }
    }
  }
  // dups before this thread's entries
  const int mine = __popc(dups);
  const int inc = warp_scan_incl(mine);
  if (lane == 31) wsum[w] = inc;
  if (!WRITE && tid == 0) sdup[kMergeThreads] = uint16_t(nA);
  __syncthreads();
  if (!WRITE) {
    if (down || i != sdup[tid + 1]) order[0] = 1;
    if (twice) order[1] = 1;
  }
  int before = inc - mine, all = 0;
#pragma unroll
  for (int v = 0; v < kMergeThreads / 32; ++v) {
    const int c = wsum[v];
    if (v < w) before += c;
    all += c;
  }
  // rows that start in this tile (the last tile: up to row m)
  const int64_t last = blockIdx.x == ntiles - 1 ? m + 1 : c1.first;
  if (!WRITE) {
    if (tid == 0) {
      tilec[blockIdx.x] = n - all;
      if (last - c0.first > kTileRows) order[2] = 1;
    }
    return;
  }
  // the inputs are dead: their space takes the output in order
  int p = x0 - before;
#pragma unroll
  for (int t = 0; t < kMergePer; ++t) {
    if (x0 + t < n && !((dups >> t) & 1u)) {
      sc[p] = col[t];
      sv[p] = val[t];
      ++p;
    }
  }
  sdup[tid] = uint16_t(before);
  sbit[tid] = uint8_t(dups);
  if (tid == 0) {
    sdup[kMergeThreads] = uint16_t(all);
    sbit[kMergeThreads] = 0;
  }
  __syncthreads();
  const int64_t o = off[blockIdx.x];
#pragma unroll
  for (int t = 0; t < kMergePer; ++t) {
    const int x = tid + t * kMergeThreads;
    if (x < n - all) {
      Cj[o + x] = sc[x];
      Cx[o + x] = sv[x];
    }
  }
  auto slot = [&](int x) {  // output entries before entry x of the tile
    return x - sdup[x / kMergePer] -
           __popc(sbit[x / kMergePer] & ((1u << (x % kMergePer)) - 1u));
  };
  if (pos) {
    for (int x = tid; x < n; x += kMergeThreads)
      pos[int64_t(blockIdx.x) * kMergeTile + x] = uint16_t(slot(x));
    return;
  }
  for (int64_t r = c0.first + tid; r < last; r += kMergeThreads) {
    const int64_t at = o + slot(int(int64_t(Ap[r]) - ab - c0.i + int64_t(Bp[r]) - bb - c0.j));
    if (cp_bits == 32) ((int32_t *)Cp)[r] = int32_t(at);
    else ((int64_t *)Cp)[r] = at;
  }
}

// strict: rows with repeated columns are refused, too.
template <typename PTA, typename PTB, typename VT>
static int spadd_impl(tspg_ctx *ctx, cudaStream_t s, const tspg_csr *A,
                      const tspg_csr *B, tspg_csr_out *C, bool strict) {
  const int64_t m = A->nrows, total = A->nnz + B->nnz;
  if (m == 0 || total == 0) {
    C->nnz = 0;
    TSPG_CUDA(ctx, cudaMemsetAsync(C->rowptr, 0, size_t(m + 1) * (C->rowptr_bits / 8), s));
    return TSPG_OK;
  }
  const int64_t ntiles = (total + kMergeTile - 1) / kMergeTile;
  const int64_t nb = (ntiles + kScanTile - 1) / kScanTile;
  Scratch sc(ctx, s);
  MergeCut *cuts;
  int32_t *tilec;
  int64_t *off, *partial;
  Sched *rec;
  TSPG_TRY(sc.get_all(part(&cuts, ntiles + 1), part(&tilec, ntiles), part(&off, ntiles + 1),
                      part(&partial, nb + 1), part(&rec, 1)));
  const PTA *Ap = (const PTA *)A->rowptr;
  const PTB *Bp = (const PTB *)B->rowptr;
  k_merge_cuts<PTA, PTB><<<unsigned((ntiles + 128) / 128), 128, 0, s>>>(m, Ap, A->col, Bp, B->col,
                                                                       ntiles, cuts, rec);
  int64_t *h = ctx->h_words;  // [0] nnz(C), [1] and [2] the order check, [3] a tile of many rows
  h[1] = h[2] = h[3] = 0;
  k_merge_tiles<false, PTA, PTB, VT><<<unsigned(ntiles), kMergeThreads, 0, s>>>(
      m, Ap, A->col, nullptr, Bp, B->col, nullptr, ntiles, cuts, tilec, h + 1, nullptr, nullptr,
      nullptr, 0, nullptr, nullptr);
  ctx->launches += 2;
  launch_scan(ctx, s, tilec, ntiles, partial, off, rec, nullptr, HostWords(), h);
  TSPG_CUDA(ctx, cudaGetLastError());
  TSPG_CUDA(ctx, cudaStreamSynchronize(s));
  const int64_t nnz = h[0];
  if (h[1] || (strict && h[2])) return TSPG_EUNSORTED;
  if (C->rowptr_bits == 32 && nnz > INT32_MAX) return TSPG_EOVERFLOW;
  TSPG_TRY(ensure_out(ctx, C, nnz, int(sizeof(VT)), s));
  // (refused by the budget: the tiles' CTAs walk their rows)
  uint16_t *pos = nullptr;
  if (h[3] && sc.get(&pos, size_t(total)) != TSPG_OK) pos = nullptr;
  k_merge_tiles<true, PTA, PTB, VT><<<unsigned(ntiles), kMergeThreads, 0, s>>>(
      m, Ap, A->col, (const VT *)A->val, Bp, B->col, (const VT *)B->val, ntiles, cuts, nullptr, nullptr, off,
      pos, C->rowptr, C->rowptr_bits, C->col, (VT *)C->val);
  ctx->launches += 1;
  if (pos) {
    k_tile_offsets<kMergeTile, PTA, PTB><<<unsigned((m + 256) / 256), 256, 0, s>>>(
        Ap, Bp, m, off, ntiles, pos, C->rowptr, C->rowptr_bits);
    ctx->launches += 1;
  }
  TSPG_CUDA(ctx, cudaGetLastError());
  return TSPG_OK;
}

int spadd_entry(tspg_ctx *ctx, void *stream, const tspg_csr *A, const tspg_csr *B, tspg_csr_out *C,
                bool strict) {
  if (!ctx || !C) return TSPG_EINVAL;
  TSPG_TRY(check_csr(A));
  TSPG_TRY(check_csr(B));
  if (A->nrows != B->nrows || A->ncols != B->ncols || A->val_bits != B->val_bits)
    return TSPG_EINVAL;
  if (!C->rowptr || C->nrows != A->nrows || C->ncols != A->ncols ||
      C->val_bits != A->val_bits || (C->rowptr_bits != 32 && C->rowptr_bits != 64))
    return TSPG_EINVAL;
  cudaStream_t s = (cudaStream_t)stream;
  TSPG_CUDA(ctx, cudaSetDevice(ctx->device));
  const int a = A->rowptr_bits, b = B->rowptr_bits;
  if (A->val_bits == 64) {
    if (a == 32 && b == 32) return spadd_impl<int32_t, int32_t, double>(ctx, s, A, B, C, strict);
    if (a == 32 && b == 64) return spadd_impl<int32_t, int64_t, double>(ctx, s, A, B, C, strict);
    if (a == 64 && b == 32) return spadd_impl<int64_t, int32_t, double>(ctx, s, A, B, C, strict);
    return spadd_impl<int64_t, int64_t, double>(ctx, s, A, B, C, strict);
  } else {
    if (a == 32 && b == 32) return spadd_impl<int32_t, int32_t, float>(ctx, s, A, B, C, strict);
    if (a == 32 && b == 64) return spadd_impl<int32_t, int64_t, float>(ctx, s, A, B, C, strict);
    if (a == 64 && b == 32) return spadd_impl<int64_t, int32_t, float>(ctx, s, A, B, C, strict);
    return spadd_impl<int64_t, int64_t, float>(ctx, s, A, B, C, strict);
  }
}

}  // namespace tspg

extern "C" int tspg_spadd(tspg_ctx *ctx, void *stream, const tspg_csr *A,
                          const tspg_csr *B, tspg_csr_out *C) {
  return tspg::spadd_entry(ctx, stream, A, B, C, false);
}
