// spgemm.cu — host side of the two-phase SpGEMM (C = A·B, C = C_in + A·B).
//
// Call sequence of one product on the caller's stream:
//   k_setup, [k_check_sorted_rows: column-window rows only], k_row_mults,
//   k_scatter<sym>, k_span / k_phase + k_groups <symbolic>, the scan, whose
//   last block leaves nnz(C), the longest A row and the class counts in mapped
//   host memory, one stream sync, then k_scatter<num>, which takes the output
//   arrays, k_dense_rank, k_span / k_phase + k_groups <numeric>.
// Products of kFuseRows rows or more spend a small launch of their own on the
// list offsets and the host's words instead of a last block.  1024 uniform
// rows of 17 entries: 24 launches, 3 copies and 8 allocations, 171 us -> 10
// launches and one allocation, 99 us.
// KokkosSparse::spgemm (include/KokkosWrap.hpp:375) and the cuSPARSE paths
// (include/cusparse_helpers.cuh:908-1344) do the same job with library-owned
// allocation and ~10 stream syncs per call.
#include <algorithm>
#include <initializer_list>
#include <new>
#include <utility>

#include "spgemm_span.cuh"

using namespace tspg;

struct tspg_plan {
  tspg_ctx *ctx = nullptr;
  cudaStream_t stream = nullptr;
  int pt_bits = 32, vt_bits = 64;
  int64_t m = 0, k = 0, n = 0;
  int64_t a_nnz = 0, b_nnz = 0;
  int64_t c_nnz = 0;
  int64_t mults = 0;
  int64_t max_a_row = 0;
  int64_t ncnt[NCLS] = {};  // numeric rows per class
  Tune tune{};                  // row binning of the symbolic call
  void *prods = nullptr;
  int64_t *base = nullptr;
  int64_t *rowf = nullptr;
  int32_t *rowc = nullptr;
  int64_t *cp = nullptr;
  uint64_t *list = nullptr;
  Sched *sched = nullptr;  // [0] symbolic, [1] numeric, [2] deferred one-pass rows
  int64_t *partial = nullptr;
  int64_t nb = 0;
  int32_t *curbuf = nullptr;
  int64_t cur_stride = 0;
  int64_t *wide_a = nullptr, *wide_b = nullptr;  // widened row offsets (mixed widths)
  tspg_csr E{};        // addend of C = E + A·B (tspg_spgemm_acc), E.col == nullptr if none
  int64_t onepass = 0;  // entries of the one-pass rows' scratch (0: none)
  int32_t *oj = nullptr;
  void *ox = nullptr;
  uint64_t *defer = nullptr;
  uint32_t *bits = nullptr;  // DENSE rows' bitmaps for the numeric phase (one-shot products)
  int32_t *slot = nullptr;
  int64_t nslots = 0, slot_words = 0;
  void *blocks[16];
  int nblocks = 0;

  template <typename T>
  int get(T **p, size_t count) {
    void *q = nullptr;
    size_t bytes = count * sizeof(T);
    if (bytes == 0) bytes = 16;
    if (nblocks == int(sizeof(blocks) / sizeof(blocks[0]))) return TSPG_ENOMEM;
    int st = ws_alloc(ctx, &q, bytes, stream);
    if (st != TSPG_OK) return st;
    blocks[nblocks++] = q;
    *p = (T *)q;
    return TSPG_OK;
  }
  // n arrays out of one block (each on a 256-byte boundary)
  int get_all(std::initializer_list<std::pair<void **, size_t>> parts) {
    size_t total = 0;
    for (auto &p : parts) total += (p.second + 255) & ~size_t(255);
    char *q = nullptr;
    TSPG_TRY(get(&q, total));
    for (auto &p : parts) {
      *p.first = q;
      q += (p.second + 255) & ~size_t(255);
    }
    return TSPG_OK;
  }
  // Give up the kept bitmaps (the numeric phase then walks those rows twice).
  void drop_bits() {
    for (void *p : {(void *)bits, (void *)slot}) {
      for (int i = 0; p && i < nblocks; ++i) {
        if (blocks[i] != p) continue;
        ws_free(ctx, p, stream);
        blocks[i] = blocks[--nblocks];
        break;
      }
    }
    bits = nullptr;
    slot = nullptr;
    nslots = 0;
  }
  ~tspg_plan() {
    for (int i = nblocks - 1; i >= 0; --i) ws_free(ctx, blocks[i], stream);
  }
};

namespace tspg {

// Internal flag of the one-shot product (tspg_spgemm): warp rows may be
// multiplied whole in the symbolic launch (one-pass rows).  A plan that is
// kept for numeric calls with new values cannot use it.
constexpr int kFlagOnePass = 1 << 30;
// ... and only on products of at least this many rows (it adds a scan and a
// host round trip before the symbolic launch), with a scratch of at most
// this many entries.
constexpr int64_t kOnePassMinRows = 1 << 16;
static_assert(kOnePassMinRows >= kFuseRows, "the one-pass branch sets the list offsets itself");
constexpr int64_t kOnePassMaxEntries = int64_t(1) << 30;

// One-shot products keep the column bitmaps of their heaviest DENSE rows from
// the symbolic to the numeric phase, which then walks those rows' products once
// instead of twice — while B's columns and values fit the L2 beside the outputs
// (beyond it the first walk is what brings B in: on R-MAT scale 20 keeping 4 GB
// of bitmaps made the numeric phase 4 % slower), in at most 4 GB of workspace,
// and for enough rows.
constexpr int64_t kKeepBytes = int64_t(4) << 30;
constexpr int64_t kKeepNnz = int64_t(6) << 20;
constexpr int64_t kKeepRows = 1024;

// Warp-class rows from which the check of B's rows for strict order pays.
constexpr int64_t kStrictRows = 4096;

static inline unsigned grid_for(int64_t work, int per_block, int cap) {
  int64_t g = (work + per_block - 1) / per_block;
  if (g < 1) g = 1;
  if (g > cap) g = cap;
  return (unsigned)g;
}

template <typename PT, typename VT>
static int symbolic_impl(tspg_ctx *ctx, cudaStream_t s, const tspg_csr *A,
                         const tspg_csr *B, int flags, tspg_plan *P) {
  TSPG_TRY(set_smem_attr<PT, VT>(ctx));
  const int64_t m = A->nrows, n = B->ncols, k = A->ncols;
  const Tune tune = P->tune = span_tune<PT, VT>(ctx->tune, n, P->E.col && P->E.nnz > 0);
  P->m = m;
  P->n = n;
  P->k = k;
  P->a_nnz = A->nnz;
  P->b_nnz = B->nnz;
  P->nb = (m + kScanTile - 1) / kScanTile;
  TSPG_TRY(P->get_all({{&P->prods, sizeof(ProdDev<PT, VT>)},
                       {(void **)&P->base, 2 * sizeof(int64_t)},
                       {(void **)&P->sched, 3 * sizeof(Sched)},
                       {(void **)&P->rowf, m * sizeof(int64_t)},
                       {(void **)&P->rowc, m * sizeof(int32_t)},
                       {(void **)&P->cp, (m + 1) * sizeof(int64_t)},
                       {(void **)&P->list, m * sizeof(uint64_t)},
                       {(void **)&P->partial, (P->nb + 1) * sizeof(int64_t)}}));
  ProdDev<PT, VT> *prods = (ProdDev<PT, VT> *)P->prods;
  bool onepass = (flags & kFlagOnePass) && !(P->E.col && P->E.nnz > 0) && m >= kOnePassMinRows;

  ProdDev<PT, VT> v{};
  v.Ap = (const PT *)A->rowptr;
  v.Aj = A->col;
  v.Ax = (const VT *)A->val;
  v.Bp = (const PT *)B->rowptr;
  v.Bj = B->col;
  v.Bx = (const VT *)B->val;
  v.m = m;
  v.n = n;
  v.cp_bits = 64;
  v.b_sorted = 1;
  if (P->E.col && P->E.nnz > 0) {
    v.Ep = P->E.rowptr;
    v.Ej = P->E.col;
    v.Ex = (const VT *)P->E.val;
    v.ep_bits = P->E.rowptr_bits;
  }
  k_setup<PT, VT><<<1, 128, 0, s>>>(prods, v, P->base, P->sched, 3, tune, onepass ? 1 : 0);
  ctx->launches += 1;
  // sorted B rows only matter to the column-window rows
  if (!(flags & TSPG_F_B_SORTED) && B->nnz > 0 && B->nrows > 0 && needs_sorted(tune, n)) {
    k_check_sorted_rows<PT><<<grid_for(B->nrows * 32, 256, ctx->num_sms * 16), 256,
                              0, s>>>(v.Bp, v.Bj, B->nrows, &prods->b_sorted);
    ctx->launches += 1;
  }
  int64_t *h = ctx->h_words;
  if (m == 0) {
    TSPG_CUDA(ctx, cudaGetLastError());
    return TSPG_OK;  // nothing to count: c_nnz, mults and max_a_row stay 0
  }
  const bool fuse = m < kFuseRows;
  launch_row_mults<PT, VT>(ctx, s, prods, P->base, 1, m, P->rowf, P->sched, P->rowc, fuse,
                           fuse ? nullptr : P->list);
  if (onepass) {
    // the one-pass rows' scratch offsets: a scan of their output bounds
    launch_scan(ctx, s, P->rowc, m, P->partial, P->cp, P->sched + 1, nullptr);
    TSPG_CUDA(ctx, cudaGetLastError());
    TSPG_CUDA(ctx, cudaMemcpyAsync(h + HW_TOTAL, P->cp + m, sizeof(int64_t),
                                   cudaMemcpyDeviceToHost, s));
    TSPG_CUDA(ctx, cudaMemcpyAsync(h + HW_CNT, &P->sched[0].cnt, NCLS * sizeof(int64_t),
                                   cudaMemcpyDeviceToHost, s));
    TSPG_CUDA(ctx, cudaStreamSynchronize(s));
    const int64_t tot = h[HW_TOTAL], rows = h[HW_CNT + CLS_ONEPASS];
    // one pass when most rows take it (R-MAT 20: a tenth of the rows, and
    // those with more than 32 outputs need their second attempt: +0.9 ms
    // of symbolic phase; Galerkin A·P: every row, -0.9 ms per call)
    if (tot > 0 && 2 * rows >= m && tot <= kOnePassMaxEntries &&
        P->get(&P->oj, size_t(tot)) == TSPG_OK && P->get((VT **)&P->ox, size_t(tot)) == TSPG_OK &&
        P->get(&P->defer, size_t(rows)) == TSPG_OK) {
      P->onepass = tot;
    } else {  // every row two-pass: the one-pass rows back to their classes
      onepass = false;
      k_fold_onepass<<<1, 32, 0, s>>>(P->sched);
      ctx->launches += 1;
    }
    // room for the bitmaps of the heaviest DENSE rows
    const int64_t dense = h[HW_CNT] + h[HW_CNT + 1] + h[HW_CNT + 2];
    const int64_t words = ((n + 1023) >> 10) * 32;
    const int64_t slots = std::min(dense, kKeepBytes / (words * 4));
    if (slots >= kKeepRows && B->nnz <= kKeepNnz && n <= kRankMaxCols && sym_dense_span<PT, VT>(n)) {
      if (P->get(&P->slot, size_t(m)) == TSPG_OK && P->get(&P->bits, size_t(slots * words)) == TSPG_OK) {
        TSPG_CUDA(ctx, cudaMemsetAsync(P->slot, 0xff, size_t(m) * sizeof(int32_t), s));
        P->nslots = slots;
        P->slot_words = words;
      } else {
        P->drop_bits();
      }
    }
  }
  if (m >= kFuseRows) {
    k_sched_offsets<<<1, 32, 0, s>>>(P->sched);
    ctx->launches += 1;
  }
  k_scatter<PT, VT, 0><<<grid_for(m, 256, INT32_MAX), 256, 0, s>>>(
      prods, P->base, 1, m, P->rowf, P->rowc, P->cp, P->sched, P->list);
  ctx->launches += 1;
  PhaseArgs pa{P->base, P->sched, P->list, P->rowf, P->rowc, P->cp,
               nullptr, 0, ctx->d_words + kErrWord, ctx->d_prof};
  pa.oj = P->oj;
  pa.ox = P->ox;
  pa.defer = P->defer;
  if (P->nslots) {
    pa.bits = P->bits;
    pa.slot = P->slot;
    pa.nslots = P->nslots;
    pa.slot_words = P->slot_words;
  }
  phase_mark(ctx, 0, 0, s);
  TSPG_TRY((launch_symbolic_rows<PT, VT>(ctx, s, prods, pa, n, true)));
  if (onepass) {
    k_lanes<false, PT, VT><<<ctx->num_sms, kOnepassThreads, kOnepassSmem, s>>>(prods, pa);
    // the rows sent back (too many columns for their 64-slot attempt and
    // too large for a warp's full table): their symbolic count, as
    // 256-thread rows of their own record
    Sched *D = P->sched + 2;
    k_defer_setup<<<1, 32, 0, s>>>(P->sched, D);
    k_sched_offsets<<<1, 32, 0, s>>>(D);
    PhaseArgs pd = pa;
    pd.S = D;
    pd.list = P->defer;
    k_groups<PT, VT, false><<<ctx->num_sms, kGroupThreads, kGroupDynSmem, s>>>(prods, pd);
    ctx->launches += 4;
  }
  phase_mark(ctx, 0, 1, s);
  HostWords sh;
  sh.words = h;
  sh.sym = P->sched;
  sh.err = ctx->d_words + kErrWord;
  launch_scan(ctx, s, P->rowc, m, P->partial, P->cp, P->sched + 1, P->rowf, sh);
  TSPG_CUDA(ctx, cudaGetLastError());
  TSPG_CUDA(ctx, cudaStreamSynchronize(s));
  P->c_nnz = h[HW_TOTAL];
  P->mults = h[HW_MULTS];
  P->max_a_row = h[HW_MAX_A];
  for (int c = 0; c < NCLS; ++c) P->ncnt[c] = h[HW_CNT + c];
  if (h[HW_ERR] != 0) {
    cudaMemsetAsync(ctx->d_words + kErrWord, 0, sizeof(int64_t), s);
    return TSPG_ECUDA;
  }
  return TSPG_OK;
}

template <typename PT, typename VT>
static int numeric_impl(tspg_ctx *ctx, cudaStream_t s, tspg_plan *P, const tspg_csr *B,
                        tspg_csr_out *C) {
  const int64_t m = P->m;
  ProdDev<PT, VT> *prods = (ProdDev<PT, VT> *)P->prods;
  if (m == 0) {
    k_set_out<PT, VT><<<1, 1, 0, s>>>(prods, C->col, (VT *)C->val, C->rowptr,
                                      C->rowptr_bits);
    k_zero_rowptr<PT, VT><<<1, 32, 0, s>>>(prods, 1);
    ctx->launches += 2;
    TSPG_CUDA(ctx, cudaGetLastError());
    return TSPG_OK;
  }
  if (P->max_a_row > kDenseCurSmem && !P->curbuf) {
    P->cur_stride = P->max_a_row;
    const size_t words = 2 * size_t(ctx->num_sms) * P->cur_stride;
    int st = P->get(&P->curbuf, words);
    if (st == TSPG_ENOMEM && P->nslots) {  // what the phase needs comes before the kept bitmaps
      P->drop_bits();
      st = P->get(&P->curbuf, words);
    }
    TSPG_TRY(st);
  }
  OutArgs out;
  out.Cj = C->col;
  out.Cx = C->val;
  out.Cp = C->rowptr;
  out.cp_bits = C->rowptr_bits;
  out.set = 1;
  out.finish = m < kFuseRows;
  if (m >= kFuseRows) {
    k_sched_offsets<<<1, 32, 0, s>>>(P->sched + 1);
    ctx->launches += 1;
  }
  // warp rows over long B rows take their span from the rows' ends, and add
  // without atomics, when B's rows are sorted and hold no column twice: worth a
  // pass over B's columns where they are many (in every call: a plan's operands
  // have one pattern, but the order inside their rows is the call's; 27-point
  // stencil on 63^3, 6.6M columns: beside the scatter, nothing of 1.64 ms)
  const bool check = !P->onepass && P->ncnt[CLS_G32] >= kStrictRows &&
                     B->nnz >= kSeqRow * B->nrows && P->mults >= 8 * B->nnz;
  if (check) {
    k_check_strict<PT, VT><<<grid_for(B->nnz, 2048, ctx->num_sms * 8), 256, 0, s>>>(
        (const PT *)B->rowptr, B->col, B->nrows, P->sched + 2, prods);
    ctx->launches += 1;
  }
  TSPG_CUDA(ctx, launch_phase(check, grid_for(m, 256, INT32_MAX), 256, 0, s, k_scatter<PT, VT, 1>,
                              prods, P->base, 1, m, P->rowf, P->rowc, P->cp, P->sched + 1, P->list,
                              out));
  PhaseArgs pa{P->base, P->sched + 1, P->list, P->rowf, P->rowc, P->cp,
               P->curbuf, P->cur_stride, ctx->d_words + kErrWord,
               ctx->d_prof ? ctx->d_prof + kProfPerPhase : nullptr};
  if (P->nslots) {
    pa.bits = P->bits;
    pa.slot = P->slot;
    pa.slot_words = P->slot_words;
  }
  phase_mark(ctx, 1, 0, s);
  TSPG_TRY((launch_numeric_rows<PT, VT>(ctx, s, prods, pa, P->n, P->tune, P->ncnt,
                                        P->c_nnz > 0 ? P->mults / P->c_nnz : 0, m < kFuseRows, true)));
  if (P->onepass)
    k_onepass_copy<PT, VT><<<grid_for(m * 32, 256, ctx->num_sms * 16), 256, 0, s>>>(
        prods, P->rowf, P->rowc, P->cp, P->oj, (const VT *)P->ox, m);
  phase_mark(ctx, 1, 1, s);
  ctx->launches += 1 + (P->onepass ? 1 : 0);
  TSPG_CUDA(ctx, cudaGetLastError());
  return TSPG_OK;
}

static int check_pair(const tspg_csr *A, const tspg_csr *B) {
  TSPG_TRY(check_csr(A));
  TSPG_TRY(check_csr(B));
  if (A->ncols != B->nrows) return TSPG_EINVAL;
  if (A->val_bits != B->val_bits) return TSPG_EINVAL;
  return TSPG_OK;
}

static int check_out(const tspg_csr_out *C, int64_t m, int64_t n, int vbits) {
  if (!C || !C->rowptr) return TSPG_EINVAL;
  if (C->nrows != m || C->ncols != n) return TSPG_EINVAL;
  if (C->rowptr_bits != 32 && C->rowptr_bits != 64) return TSPG_EINVAL;
  if (C->val_bits != vbits) return TSPG_EINVAL;
  return TSPG_OK;
}

template <typename F>
static int dispatch(int pt_bits, int vt_bits, F &&f) {
  if (pt_bits == 32 && vt_bits == 64) return f((int32_t *)0, (double *)0);
  if (pt_bits == 64 && vt_bits == 64) return f((int64_t *)0, (double *)0);
  if (pt_bits == 32 && vt_bits == 32) return f((int32_t *)0, (float *)0);
  if (pt_bits == 64 && vt_bits == 32) return f((int64_t *)0, (float *)0);
  return TSPG_EINVAL;
}

}  // namespace tspg

extern "C" int tspg_plan_destroy(tspg_plan *plan) {
  if (!plan) return TSPG_EINVAL;
  cudaSetDevice(plan->ctx->device);
  delete plan;
  return TSPG_OK;
}

static int plan_get(tspg_ctx *, void *plan, int64_t **p, int64_t n) {
  return ((tspg_plan *)plan)->get(p, size_t(n));
}

// Symbolic phase of A·B, or of E + A·B when E is given (its entries join
// their rows as products with coefficient 1).
static int symbolic_entry(tspg_ctx *ctx, void *stream, const tspg_csr *A_in,
                          const tspg_csr *B_in, const tspg_csr *E, int flags,
                          tspg_plan **plan, int64_t *c_nnz) {
  if (!ctx || !plan) return TSPG_EINVAL;
  *plan = nullptr;
  TSPG_TRY(check_pair(A_in, B_in));
  cudaStream_t s = (cudaStream_t)stream;
  TSPG_CUDA(ctx, cudaSetDevice(ctx->device));
  tspg_plan *P = new (std::nothrow) tspg_plan();
  if (!P) return TSPG_ENOMEM;
  P->ctx = ctx;
  P->stream = s;
  if (E) P->E = *E;
  tspg_csr a = *A_in, b = *B_in;
  const tspg_csr *A = &a, *B = &b;
  if (a.rowptr_bits != b.rowptr_bits) {
    tspg_csr *M = a.rowptr_bits == 32 ? &a : &b;
    int64_t **buf = M == &a ? &P->wide_a : &P->wide_b;
    int st = P->get(buf, size_t(M->nrows + 1));
    if (st != TSPG_OK) {
      delete P;
      return st;
    }
    k_widen<<<(unsigned)((M->nrows + 1 + 255) / 256), 256, 0, s>>>((const int32_t *)M->rowptr,
                                                                    M->nrows + 1, *buf);
    ctx->launches += 1;
    M->rowptr = *buf;
    M->rowptr_bits = 64;
  }
  P->pt_bits = A->rowptr_bits;
  P->vt_bits = A->val_bits;
  int st = dispatch(P->pt_bits, P->vt_bits, [&](auto pt, auto vt) {
    using PT = std::remove_pointer_t<decltype(pt)>;
    using VT = std::remove_pointer_t<decltype(vt)>;
    return symbolic_impl<PT, VT>(ctx, s, A, B, flags, P);
  });
  if (st != TSPG_OK) {
    delete P;
    return st;
  }
  if (c_nnz) *c_nnz = P->c_nnz;
  *plan = P;
  return TSPG_OK;
}

extern "C" int tspg_spgemm_symbolic(tspg_ctx *ctx, void *stream,
                                    const tspg_csr *A_in, const tspg_csr *B_in,
                                    int flags, tspg_plan **plan,
                                    int64_t *c_nnz) {
  return symbolic_entry(ctx, stream, A_in, B_in, nullptr, flags, plan, c_nnz);
}

extern "C" int tspg_spgemm_numeric(tspg_ctx *ctx, void *stream,
                                   tspg_plan *plan, const tspg_csr *A_in,
                                   const tspg_csr *B_in, tspg_csr_out *C) {
  if (!ctx || !plan) return TSPG_EINVAL;
  TSPG_TRY(check_pair(A_in, B_in));
  tspg_csr a = *A_in, b = *B_in;
  const tspg_csr *A = &a, *B = &b;
  if (a.rowptr_bits != b.rowptr_bits) {
    tspg_csr *M = a.rowptr_bits == 32 ? &a : &b;
    int64_t *buf = M == &a ? plan->wide_a : plan->wide_b;
    if (!buf) return TSPG_EINVAL;  // the symbolic call had matching widths
    k_widen<<<(unsigned)((M->nrows + 1 + 255) / 256), 256, 0, (cudaStream_t)stream>>>(
        (const int32_t *)M->rowptr, M->nrows + 1, buf);
    ctx->launches += 1;
    M->rowptr = buf;
    M->rowptr_bits = 64;
  }
  if (A->nrows != plan->m || B->ncols != plan->n || A->nnz != plan->a_nnz ||
      B->nnz != plan->b_nnz || A->rowptr_bits != plan->pt_bits ||
      A->val_bits != plan->vt_bits)
    return TSPG_EINVAL;
  TSPG_TRY(check_out(C, plan->m, plan->n, plan->vt_bits));
  if (C->rowptr_bits == 32 && plan->c_nnz > INT32_MAX) return TSPG_EOVERFLOW;
  cudaStream_t s = (cudaStream_t)stream;
  TSPG_CUDA(ctx, cudaSetDevice(ctx->device));
  TSPG_TRY(ensure_out(ctx, C, plan->c_nnz, plan->vt_bits / 8, s));
  // the plan's prods descriptor points at the symbolic call's operands; the
  // numeric call may pass new value arrays of the same pattern
  return dispatch(plan->pt_bits, plan->vt_bits, [&](auto pt, auto vt) {
    using PT = std::remove_pointer_t<decltype(pt)>;
    using VT = std::remove_pointer_t<decltype(vt)>;
    ProdDev<PT, VT> v{};
    v.Ap = (const PT *)A->rowptr;
    v.Aj = A->col;
    v.Ax = (const VT *)A->val;
    v.Bp = (const PT *)B->rowptr;
    v.Bj = B->col;
    v.Bx = (const VT *)B->val;
    v.m = A->nrows;
    v.n = B->ncols;
    v.cp_bits = 64;
    ProdDev<PT, VT> *prods = (ProdDev<PT, VT> *)plan->prods;
    k_set_operands<PT, VT><<<1, 1, 0, s>>>(prods, v);
    ctx->launches += 1;
    return numeric_impl<PT, VT>(ctx, s, plan, B, C);
  });
}

extern "C" int tspg_spgemm(tspg_ctx *ctx, void *stream, const tspg_csr *A,
                           const tspg_csr *B, tspg_csr_out *C, int flags) {
  if (!ctx) return TSPG_EINVAL;
  TSPG_TRY(check_pair(A, B));
  TSPG_TRY(check_out(C, A->nrows, B->ncols, A->val_bits));
  tspg_plan *plan = nullptr;
  int64_t nnz = 0;
  TSPG_TRY(symbolic_entry(ctx, stream, A, B, nullptr, (flags & ~kFlagOnePass) | kFlagOnePass, &plan,
                          &nnz));
  int st = TSPG_OK;
  if (C->rowptr_bits == 32 && nnz > INT32_MAX) st = TSPG_EOVERFLOW;
  OutBlocks got;
  if (st == TSPG_OK) st = ensure_out(ctx, C, nnz, A->val_bits / 8, (cudaStream_t)stream, &got);
  if (st == TSPG_ENOMEM && C->alloc && plan->nslots) {
    // the output comes before the kept bitmaps
    plan->drop_bits();
    st = ensure_out(ctx, C, nnz, A->val_bits / 8, (cudaStream_t)stream, &got);
  }
  if (st == TSPG_OK) {
    st = dispatch(plan->pt_bits, plan->vt_bits, [&](auto pt, auto vt) {
      using PT = std::remove_pointer_t<decltype(pt)>;
      using VT = std::remove_pointer_t<decltype(vt)>;
      // B with the offsets the symbolic phase used (widened when mixed)
      tspg_csr b = *B;
      if (plan->wide_b) b.rowptr = plan->wide_b;
      return numeric_impl<PT, VT>(ctx, (cudaStream_t)stream, plan, &b, C);
    });
  }
  tspg_plan_destroy(plan);
  return st;
}

extern "C" int tspg_spgemm_count(tspg_ctx *ctx, void *stream,
                                 const tspg_csr *A, const tspg_csr *B,
                                 int64_t *mults, int64_t *c_nnz_upper) {
  if (!ctx) return TSPG_EINVAL;
  TSPG_TRY(check_pair(A, B));
  cudaStream_t s = (cudaStream_t)stream;
  TSPG_CUDA(ctx, cudaSetDevice(ctx->device));
  Scratch sc(ctx, s);
  tspg_csr a = *A, b = *B;
  if (a.rowptr_bits != b.rowptr_bits) {
    tspg_csr *M = a.rowptr_bits == 32 ? &a : &b;
    int64_t *buf;
    TSPG_TRY(sc.get(&buf, M->nrows + 1));
    k_widen<<<(unsigned)((M->nrows + 1 + 255) / 256), 256, 0, s>>>((const int32_t *)M->rowptr,
                                                                    M->nrows + 1, buf);
    ctx->launches += 1;
    M->rowptr = buf;
    M->rowptr_bits = 64;
  }
  A = &a;
  B = &b;
  return dispatch(A->rowptr_bits, A->val_bits, [&](auto pt, auto vt) -> int {
    using PT = std::remove_pointer_t<decltype(pt)>;
    using VT = std::remove_pointer_t<decltype(vt)>;
    const int64_t m = A->nrows;
    ProdDev<PT, VT> *prods;
    int64_t *base, *rowf;
    Sched *sched;
    TSPG_TRY(sc.get(&prods, 1));
    TSPG_TRY(sc.get(&base, 2));
    TSPG_TRY(sc.get(&rowf, m));
    TSPG_TRY(sc.get(&sched, 1));
    ProdDev<PT, VT> v{};
    v.Ap = (const PT *)A->rowptr;
    v.Aj = A->col;
    v.Bp = (const PT *)B->rowptr;
    v.m = m;
    v.n = B->ncols;
    k_setup<PT, VT><<<1, 128, 0, s>>>(prods, v, base, sched, 1, ctx->tune, 0);
    if (m > 0)
      launch_row_mults<PT, VT>(ctx, s, prods, base, 1, m, rowf, sched, nullptr, 0, nullptr);
    ctx->launches += 1;
    TSPG_CUDA(ctx, cudaGetLastError());
    int64_t *h = ctx->h_words;
    TSPG_CUDA(ctx, cudaMemcpyAsync(h, &sched->total, 2 * sizeof(int64_t),
                                   cudaMemcpyDeviceToHost, s));
    TSPG_CUDA(ctx, cudaStreamSynchronize(s));
    if (mults) *mults = h[0];
    if (c_nnz_upper) *c_nnz_upper = h[1];
    return TSPG_OK;
  });
}

namespace tspg {

// Flop count of A·B fused with the SUMMA stage mask, over A's entries in runs
// of kMaskRun per warp (balanced however they cluster in rows; a warp per row
// waited on the hub rows of an R-MAT tile: 143 -> 62 us for 0.76M entries,
// the whole call 192 -> 112).
// Entry (i, k) adds nnz(B row k) to row i's products — summed over the lanes of
// the row, one reduction per row and window — and, when that row of B is
// non-empty, sets bit k of the word mask.  Bit k ends up set exactly when
// column k of A holds an entry and row k of B is non-empty, i.e. the AND of the
// column mask of A and the row mask of B.
constexpr int kMaskRun = 128;
template <typename APT, typename BPT>
__global__ void __launch_bounds__(256)
    k_count_mask(const APT *__restrict__ Ap, const int32_t *__restrict__ Aj,
                 const BPT *__restrict__ Bp, int64_t m, uint32_t *mask,
                 unsigned long long *rowf) {
  constexpr int U = kMaskRun / 32;
  const int lane = threadIdx.x & 31;
  const int64_t e0 = ((int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5) * kMaskRun;
  const int64_t base = int64_t(Ap[0]), count = int64_t(Ap[m]) - base;
  if (e0 >= count) return;
  int32_t k[U];
  int64_t len[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const int64_t e = e0 + u * 32 + lane;
    k[u] = e < count ? __ldg(Aj + base + e) : -1;
  }
#pragma unroll
  for (int u = 0; u < U; ++u) len[u] = k[u] >= 0 ? int64_t(__ldg(Bp + k[u] + 1)) - int64_t(__ldg(Bp + k[u])) : 0;
#pragma unroll
  for (int u = 0; u < U; ++u) {
    if (len[u] > 0) {
      const uint32_t bit = 1u << (k[u] & 31);
      if (!(*(volatile uint32_t *)(mask + (k[u] >> 5)) & bit)) atomicOr(mask + (k[u] >> 5), bit);
    }
  }
  int64_t r = first_row(Ap, m, base, e0, lane);
#pragma unroll
  for (int u = 0; u < U; ++u) {
    if (e0 + u * 32 < count) {  // uniform
      const int64_t row = window_row(Ap, m, base, r, e0 + u * 32 + lane, lane);
      // inclusive sums inside runs of one row; the run's last lane adds it
      const int64_t prev = __shfl_up_sync(0xffffffffu, row, 1);
      const unsigned heads = __ballot_sync(0xffffffffu, lane == 0 || prev != row);
      const int head = 31 - __clz(heads & (0xffffffffu >> (31 - lane)));
      int64_t sum = len[u];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int64_t x = __shfl_up_sync(0xffffffffu, sum, o);
        if (lane - o >= head) sum += x;
      }
      const bool last = lane == 31 || ((heads >> (lane + 1)) & 1u);
      if (last && sum > 0) atomicAdd(rowf + row, (unsigned long long)sum);
    }
  }
}

// Totals of the row products: mults and sum of min(products, n).
// (host: mapped memory, written by the last block)
__global__ void __launch_bounds__(256)
    k_count_totals(const unsigned long long *rowf, int64_t m, int64_t n, unsigned long long *tot,
                   uint32_t *ticket, int64_t *host) {
  unsigned long long wm = 0, wu = 0;
  const int64_t stride = int64_t(gridDim.x) * blockDim.x;
  for (int64_t r = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; r < m; r += stride) {
    const unsigned long long f = rowf[r];
    wm += f;
    wu += f < (unsigned long long)n ? f : (unsigned long long)n;
  }
  wm = warp_sum(wm);
  wu = warp_sum(wu);
  if ((threadIdx.x & 31) == 0 && (wm | wu)) {
    atomicAdd(tot, wm);
    atomicAdd(tot + 1, wu);
  }
  if (last_block(ticket) && threadIdx.x == 0) {
    volatile int64_t *h = host;
    h[0] = *(volatile int64_t *)tot;
    h[1] = *(volatile int64_t *)(tot + 1);
    __threadfence_system();
  }
}

// Word mask -> LSB-first byte mask: byte i holds bits k = 8i .. 8i + 7.
__global__ void k_mask_bytes(const uint32_t *w, int64_t nbytes, uint8_t *out) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i < nbytes) out[i] = uint8_t(w[i >> 2] >> ((i & 3) * 8));
}

template <typename APT, typename BPT>
static void launch_count_mask(tspg_ctx *ctx, cudaStream_t s, const tspg_csr *A, const tspg_csr *B,
                              uint32_t *words, unsigned long long *rowf, unsigned long long *tot) {
  if (A->nnz > 0)
    k_count_mask<APT, BPT><<<unsigned((A->nnz + 8 * kMaskRun - 1) / (8 * kMaskRun)), 256, 0, s>>>(
        (const APT *)A->rowptr, A->col, (const BPT *)B->rowptr, A->nrows, words, rowf);
  k_count_totals<<<grid_for(A->nrows, 256, ctx->num_sms * 4), 256, 0, s>>>(
      rowf, A->nrows, B->ncols, tot, (uint32_t *)(tot + 2), ctx->h_words);
  ctx->launches += 1 + (A->nnz > 0);
}

}  // namespace tspg

extern "C" int tspg_spgemm_count_mask(tspg_ctx *ctx, void *stream, const tspg_csr *A,
                                      const tspg_csr *B, uint8_t *mask, int64_t *mults,
                                      int64_t *c_nnz_upper) {
  if (!ctx) return TSPG_EINVAL;
  TSPG_TRY(check_pair(A, B));
  const int64_t kdim = A->ncols, nbytes = (kdim + 7) / 8;
  if (nbytes > 0 && !mask) return TSPG_EINVAL;
  cudaStream_t s = (cudaStream_t)stream;
  TSPG_CUDA(ctx, cudaSetDevice(ctx->device));
  Scratch sc(ctx, s);
  uint32_t *words;  // the mask words, then (8-byte aligned) two totals and the row products
  const int64_t nw = ((kdim + 31) / 32 + 1) & ~int64_t(1);
  TSPG_TRY(sc.get(&words, nw + 2 * (A->nrows + 3)));
  unsigned long long *tot = (unsigned long long *)(words + nw), *rowf = tot + 3;  // ticket between
  const int64_t zero = nw / 2 + A->nrows + 3;
  k_zero<<<grid_for(zero, 256, ctx->num_sms * 8), 256, 0, s>>>((uint64_t *)words, zero);
  ctx->launches += 1;
  if (A->nrows > 0) {
    if (A->rowptr_bits == 32 && B->rowptr_bits == 32) launch_count_mask<int32_t, int32_t>(ctx, s, A, B, words, rowf, tot);
    else if (A->rowptr_bits == 32) launch_count_mask<int32_t, int64_t>(ctx, s, A, B, words, rowf, tot);
    else if (B->rowptr_bits == 32) launch_count_mask<int64_t, int32_t>(ctx, s, A, B, words, rowf, tot);
    else launch_count_mask<int64_t, int64_t>(ctx, s, A, B, words, rowf, tot);
  }
  if (nbytes > 0) {
    k_mask_bytes<<<(unsigned)((nbytes + 255) / 256), 256, 0, s>>>(words, nbytes, mask);
    ctx->launches += 1;
  }
  TSPG_CUDA(ctx, cudaGetLastError());
  int64_t *h = ctx->h_words;
  if (A->nrows == 0) h[0] = h[1] = 0;
  TSPG_CUDA(ctx, cudaStreamSynchronize(s));
  if (mults) *mults = h[0];
  if (c_nnz_upper) *c_nnz_upper = h[1];
  return TSPG_OK;
}

// C_out = C_in + A·B: the product goes to pool workspace, then the union merge
// writes C_out (sp_mma_hybrid, include/cusparse_helpers.cuh:708-739, does the
// same with KokkosKernels + csrgeam2).
extern "C" int tspg_spgemm_acc(tspg_ctx *ctx, void *stream, const tspg_csr *A,
                               const tspg_csr *B, const tspg_csr *C_in,
                               tspg_csr_out *C_out, int flags) {
  if (!ctx) return TSPG_EINVAL;
  TSPG_TRY(check_pair(A, B));
  const bool have_in = C_in && C_in->nnz > 0;
  const int pflags = flags & TSPG_F_B_SORTED;
  if (!have_in) return tspg_spgemm(ctx, stream, A, B, C_out, pflags);
  TSPG_TRY(check_csr(C_in));
  if (C_in->nrows != A->nrows || C_in->ncols != B->ncols ||
      C_in->val_bits != A->val_bits)
    return TSPG_EINVAL;
  TSPG_TRY(check_out(C_out, A->nrows, B->ncols, A->val_bits));
  const bool fuse = (flags & TSPG_F_ACC_FUSE) ||
                    (!(flags & TSPG_F_ACC_SPLIT) && C_in->nnz <= A->nnz + B->nnz);
  // one SpGEMM in which C_in's entries join their rows as products with
  // coefficient 1
  auto fused = [&]() -> int {
    tspg_plan *plan = nullptr;
    TSPG_TRY(symbolic_entry(ctx, stream, A, B, C_in, pflags, &plan, nullptr));
    const int st = tspg_spgemm_numeric(ctx, stream, plan, A, B, C_out);
    tspg_plan_destroy(plan);
    return st;
  };
  if (fuse) return fused();
  // the product into workspace, then the merge into C_out
  cudaStream_t s = (cudaStream_t)stream;
  tspg_plan *plan = nullptr;
  int64_t nnz = 0;
  TSPG_TRY(tspg_spgemm_symbolic(ctx, stream, A, B, pflags, &plan, &nnz));
  const int vb = A->val_bits / 8;
  const int pb = nnz > INT32_MAX ? 64 : C_in->rowptr_bits;
  void *rp = nullptr, *cj = nullptr, *cx = nullptr;
  int st = ws_alloc(ctx, &rp, size_t(A->nrows + 1) * (pb / 8), s);
  if (st == TSPG_OK) st = ws_alloc(ctx, &cj, size_t(nnz > 0 ? nnz : 1) * 4, s);
  if (st == TSPG_OK) st = ws_alloc(ctx, &cx, size_t(nnz > 0 ? nnz : 1) * vb, s);
  tspg_csr_out T{};
  if (st == TSPG_OK) {
    T.nrows = A->nrows;
    T.ncols = B->ncols;
    T.rowptr = rp;
    T.rowptr_bits = pb;
    T.val_bits = A->val_bits;
    T.col = (int32_t *)cj;
    T.val = cx;
    T.capacity = nnz;
    st = tspg_spgemm_numeric(ctx, stream, plan, A, B, &T);
  }
  tspg_plan_destroy(plan);
  if (st == TSPG_OK) {
    tspg_csr prod{T.nrows, T.ncols, T.nnz, T.rowptr, T.rowptr_bits, T.val_bits,
                  T.col, T.val};
    st = spadd_entry(ctx, stream, &prod, C_in, C_out, true);
  }
  ws_free(ctx, cx, s);
  ws_free(ctx, cj, s);
  ws_free(ctx, rp, s);
  // rows of C_in in no order, or with a column twice: the merge takes neither
  return st == TSPG_EUNSORTED ? fused() : st;
}
