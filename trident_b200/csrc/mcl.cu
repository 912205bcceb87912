// mcl.cu — the per-iteration matrix updates of Markov clustering on the device.
//
// The reference's MCL driver (src/mcl.cu:56-149) copies its tile to the host
// for each of prune, normalize and inflation, loops over the rows there and
// copies the result back.  Here each is one or a few kernels on the caller's
// stream: normalize and inflation rewrite the values in place (a warp or a CTA
// per row: its sum, then the scaled values), prune compacts the kept entries
// into a new CSR (count pass, device scan, order-preserving fill).  The row sums
// are over this tile's rows only: the reference then adds the partial sums of
// the ranks of a process row (MPI_Allreduce on the row communicator), a step
// that does not exist on one GPU.
#include "spgemm_kernels.cuh"

namespace tspg {

// Rows scaled to sum 1 (entries of a row whose sum is <= 1e-20 become 0),
// after raising every value to `power` when do_pow (inflation).  Rows of up to
// 256 entries stay in a warp's registers, of up to 2048 in the CTA's: one read
// and one write of the values.  Longer ones are powered and summed, then read
// back.  The 8 rows of a CTA lie ngroups apart, so the neighbouring hub rows of
// a graph go to different CTAs (a warp per row, hub rows of 25k entries: 0.61
// ms for 46M entries).  A warp takes 32 rows, marking the long ones, before the
// CTA takes those together: meeting after every row cost matrices of short rows
// more than the reads (1M rows of 4 entries 590 -> 240 us; a warp per row 416).
// power 2 is one multiplication (pow costs ~150 instructions an entry).
template <typename VT>
__device__ __forceinline__ VT mcl_pow(VT v, VT power, int do_pow) {
  return do_pow == 2 ? v * v : do_pow ? VT(pow(v, power)) : v;
}

// One row of at most 32 U entries by one warp.
template <int U, typename VT>
__device__ __forceinline__ void mcl_warp_row(const VT *val, VT *out, int len, int lane, VT power,
                                             int do_pow) {
  VT v[U], sum = VT(0);
#pragma unroll
  for (int u = 0; u < U; ++u) v[u] = u * 32 + lane < len ? val[u * 32 + lane] : VT(0);
#pragma unroll
  for (int u = 0; u < U; ++u)
    if (u * 32 + lane < len) {
      v[u] = mcl_pow(v[u], power, do_pow);
      sum += v[u];
    }
  sum = warp_sum(sum);
  const bool keep = sum > VT(1e-20);
#pragma unroll
  for (int u = 0; u < U; ++u)
    if (u * 32 + lane < len) out[u * 32 + lane] = keep ? v[u] / sum : VT(0);
}

template <typename PT, typename VT>
__global__ void __launch_bounds__(256)
    k_mcl_rows(const PT *rp, const VT *val, int64_t m, int64_t ngroups, VT power, int do_pow,
               VT *out) {
  constexpr int U = 8;
  __shared__ VT part[8];
  __shared__ unsigned longs[8];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int64_t step = gridDim.x;
  for (int64_t g0 = blockIdx.x; g0 < ngroups; g0 += 32 * step) {
    unsigned mine = 0;
    // lane l holds the bounds of the warp's l-th row of the 32
    const int64_t gl = g0 + lane * step, rl = w * ngroups + gl;
    const bool have = gl < ngroups && rl < m;
    const int64_t s0 = have ? int64_t(rp[rl]) : 0;
    const int64_t n0 = have ? int64_t(rp[rl + 1]) - s0 : 0;
    for (unsigned todo = __ballot_sync(0xffffffffu, n0 > 0); todo; todo &= todo - 1) {
      const int t = __ffs(todo) - 1;
      const int64_t a0 = __shfl_sync(0xffffffffu, s0, t), len = __shfl_sync(0xffffffffu, n0, t);
      if (len <= 32) mcl_warp_row<1>(val + a0, out + a0, int(len), lane, power, do_pow);
      else if (len <= 32 * U) mcl_warp_row<U>(val + a0, out + a0, int(len), lane, power, do_pow);
      else mine |= 1u << t;
    }
    if (lane == 0) longs[w] = mine;
    // the longer ones, a CTA each (uniform over the CTA)
    if (!__syncthreads_or(mine != 0)) continue;
    for (int q = 0; q < 8; ++q) {
      for (unsigned todo = longs[q]; todo; todo &= todo - 1) {
        const int64_t row = q * ngroups + g0 + (__ffs(todo) - 1) * step;
        const int64_t b0 = int64_t(rp[row]), n = int64_t(rp[row + 1]) - b0;
        const bool held = n <= 256 * U;
        VT v[U], sum = VT(0);
        for (int64_t c = 0; c < n; c += 256 * U) {
#pragma unroll
          for (int u = 0; u < U; ++u) v[u] = c + u * 256 + tid < n ? val[b0 + c + u * 256 + tid] : VT(0);
#pragma unroll
          for (int u = 0; u < U; ++u)
            if (c + u * 256 + tid < n) {
              v[u] = mcl_pow(v[u], power, do_pow);
              sum += v[u];
              if (!held && do_pow) out[b0 + c + u * 256 + tid] = v[u];
            }
        }
        sum = warp_sum(sum);
        if (lane == 0) part[w] = sum;
        __syncthreads();
        sum = VT(0);
#pragma unroll
        for (int k = 0; k < 8; ++k) sum += part[k];
        const bool keep = sum > VT(1e-20);
        const VT *src = do_pow ? out : val;  // the thread's own writes, if powered
        for (int64_t c = 0; c < n; c += 256 * U) {
          if (!held) {
#pragma unroll
            for (int u = 0; u < U; ++u) v[u] = c + u * 256 + tid < n ? src[b0 + c + u * 256 + tid] : VT(0);
          }
#pragma unroll
          for (int u = 0; u < U; ++u)
            if (c + u * 256 + tid < n) out[b0 + c + u * 256 + tid] = keep ? v[u] / sum : VT(0);
        }
        __syncthreads();  // part is free again
      }
    }
    __syncthreads();  // longs is free again
  }
}

// Prune: the entries with |v| > tol, in their order.  Tiles of kPruneTile
// entries whatever the rows' lengths (a warp per row took 0.23 + 0.38 ms for
// 46M entries in rows of up to 25k); warp w of a tile owns 256 consecutive
// ones.  FILL = false leaves the tile's number of kept entries in tilec, and
// *many = 1 when two row starts kTileRows rows apart lie in one tile;
// FILL = true writes them from off[tile] on, and the offsets of the rows that
// start in the tile (pos given: the entries' slots, for k_tile_offsets).
constexpr int kPruneTile = 2048;
template <bool FILL, typename PT, typename VT>
__global__ void __launch_bounds__(256)
    k_prune_tiles(const PT *__restrict__ rp, const int32_t *__restrict__ col,
                  const VT *__restrict__ val, int64_t m, int64_t nnz, VT tol, int64_t ntiles,
                  int32_t *tilec, Sched *rec, volatile int64_t *many, const int64_t *off,
                  uint16_t *pos, void *np, int np_bits, int32_t *ocol, VT *oval) {
  constexpr int U = 8;
  __shared__ unsigned mask[64 + 1];
  __shared__ int before[64 + 1];
  __shared__ int64_t row0[2];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int64_t base = int64_t(rp[0]);
  const int64_t span = int64_t(rp[m]) - base, total = span < nnz ? span : nnz;
  const int64_t t = blockIdx.x, d0 = t * kPruneTile < total ? t * kPruneTile : total;
  const int64_t d1 = d0 + kPruneTile < total ? d0 + kPruneTile : total;
  VT v[U];
  int32_t c[U];
  unsigned b[U];
  int kept = 0;
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const int64_t e = d0 + w * 256 + u * 32 + lane;
    v[u] = e < d1 ? __ldg(val + base + e) : VT(0);
    if (FILL) c[u] = e < d1 ? __ldg(col + base + e) : 0;
  }
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const int64_t e = d0 + w * 256 + u * 32 + lane;
    b[u] = __ballot_sync(0xffffffffu, e < d1 && fabs(v[u]) > tol);
    if (lane == 0) mask[w * U + u] = b[u];
    kept += __popc(b[u]);
  }
  if (FILL && w < 2 && !pos) {
    // the first row that starts at or after d0 (w = 0), and the one that ends
    // this tile's rows (the last tile: one past row m)
    const int64_t d = w == 0 ? d0 : d1;
    int64_t lo = 0, hi = m + 1;  // rows below lo start before d, row hi does not
    while (hi > lo) {
      const int64_t step = (hi - lo + 31) / 32, i = lo + lane * step;
      const unsigned s = __ballot_sync(0xffffffffu, i < hi && int64_t(__ldg(rp + i)) - base < d);
      const int n = __popc(s);
      if (n == 0) break;
      const int64_t at = lo + int64_t(n - 1) * step;
      lo = at + 1;
      hi = at + step < hi ? at + step : hi;
    }
    if (lane == 0) row0[w] = w == 1 && t == ntiles - 1 ? m + 1 : lo;
  }
  __syncthreads();
  if (w == 0) {  // entries kept before each window of 32
    const int a = __popc(mask[2 * lane]), z = __popc(mask[2 * lane + 1]);
    const int inc = warp_scan_incl(a + z);
    before[2 * lane] = inc - a - z;
    before[2 * lane + 1] = inc - z;
    if (lane == 31) {
      before[64] = inc;
      mask[64] = 0;
    }
  }
  __syncthreads();
  if (!FILL) {
    if (tid == 0) tilec[t] = before[64];
    if (tid == 0 && t == 0) rec->ticket = 0;  // of the scan to come
    auto tile = [&](int64_t r) {
      const int64_t x = (int64_t(__ldg(rp + r)) - base) / kPruneTile;
      return x < ntiles ? x : ntiles - 1;
    };
    for (int64_t r = (t * 256 + tid) * kTileRows; r + kTileRows <= m; r += ntiles * 256 * kTileRows)
      if (tile(r) == tile(r + kTileRows)) *many = 1;
    return;
  }
  const int64_t o = off[t];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    if ((b[u] >> lane) & 1u) {
      const int64_t q = o + before[w * U + u] + __popc(b[u] & ((1u << lane) - 1u));
      ocol[q] = c[u];
      oval[q] = v[u];
    }
  }
  if (pos) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t e = d0 + w * 256 + u * 32 + lane;
      if (e < d1) pos[e] = uint16_t(before[w * U + u] + __popc(b[u] & ((1u << lane) - 1u)));
    }
    return;
  }
  for (int64_t r = row0[0] + tid; r < row0[1]; r += 256) {
    const int x = int(int64_t(__ldg(rp + r)) - base - d0);
    const int64_t q = o + before[x >> 5] + __popc(mask[x >> 5] & ((1u << (x & 31)) - 1u));
    if (np_bits == 32) ((int32_t *)np)[r] = int32_t(q);
    else ((int64_t *)np)[r] = q;
  }
}

template <typename PT, typename VT>
static int mcl_rows_impl(tspg_ctx *ctx, cudaStream_t s, const tspg_csr *M, double power,
                         int do_pow, void *val_out) {
  if (M->nrows > 0 && M->nnz > 0) {
    const int64_t ngroups = (M->nrows + 7) / 8;
    k_mcl_rows<PT, VT><<<unsigned(std::min<int64_t>(ngroups, int64_t(ctx->num_sms) * 8)), 256, 0, s>>>(
        (const PT *)M->rowptr, (const VT *)M->val, M->nrows, ngroups, VT(power),
        do_pow && power == 2.0 ? 2 : do_pow, (VT *)val_out);
    ctx->launches += 1;
  }
  TSPG_CUDA(ctx, cudaGetLastError());
  return TSPG_OK;
}

template <typename PT, typename VT>
static int prune_impl(tspg_ctx *ctx, cudaStream_t s, const tspg_csr *M, double tol,
                      tspg_csr_out *out) {
  const int64_t m = M->nrows;
  if (m == 0 || M->nnz == 0) {
    out->nnz = 0;
    TSPG_CUDA(ctx, cudaMemsetAsync(out->rowptr, 0, size_t(m + 1) * (out->rowptr_bits / 8), s));
    return TSPG_OK;
  }
  const int64_t ntiles = (M->nnz + kPruneTile - 1) / kPruneTile;
  Scratch sc(ctx, s);
  int32_t *tilec;
  int64_t *off, *partial;
  Sched *rec;
  TSPG_TRY(sc.get_all(part(&tilec, ntiles), part(&off, ntiles + 1),
                      part(&partial, (ntiles + kScanTile - 1) / kScanTile + 1), part(&rec, 1)));
  int64_t *h = ctx->h_words;  // [0] kept entries, [1] a tile of many rows
  h[1] = 0;
  k_prune_tiles<false, PT, VT><<<unsigned(ntiles), 256, 0, s>>>(
      (const PT *)M->rowptr, nullptr, (const VT *)M->val, m, M->nnz, VT(tol), ntiles, tilec, rec,
      h + 1, nullptr, nullptr, nullptr, 0, nullptr, nullptr);
  ctx->launches += 1;
  launch_scan(ctx, s, tilec, ntiles, partial, off, rec, nullptr, HostWords(), h);
  TSPG_CUDA(ctx, cudaGetLastError());
  TSPG_CUDA(ctx, cudaStreamSynchronize(s));
  const int64_t nnz = h[0];
  out->nnz = nnz;
  if (out->rowptr_bits == 32 && nnz > INT32_MAX) return TSPG_EOVERFLOW;
  TSPG_TRY(ensure_out(ctx, out, nnz, int(sizeof(VT)), s));
  // (refused by the budget: the tiles' CTAs walk their rows)
  uint16_t *pos = nullptr;
  if (h[1] && sc.get(&pos, size_t(M->nnz)) != TSPG_OK) pos = nullptr;
  k_prune_tiles<true, PT, VT><<<unsigned(ntiles), 256, 0, s>>>(
      (const PT *)M->rowptr, M->col, (const VT *)M->val, m, M->nnz, VT(tol), ntiles, nullptr, nullptr,
      nullptr, off, pos, out->rowptr, out->rowptr_bits, out->col, (VT *)out->val);
  ctx->launches += 1;
  if (pos) {
    k_tile_offsets<kPruneTile, PT, PT><<<unsigned((m + 256) / 256), 256, 0, s>>>(
        (const PT *)M->rowptr, (const PT *)nullptr, m, off, ntiles, pos, out->rowptr, out->rowptr_bits);
    ctx->launches += 1;
  }
  TSPG_CUDA(ctx, cudaGetLastError());
  return TSPG_OK;
}

}  // namespace tspg

using namespace tspg;

static int mcl_rows(tspg_ctx *ctx, void *stream, const tspg_csr *M, double power, int do_pow,
                    void *val_out) {
  if (!ctx) return TSPG_EINVAL;
  TSPG_TRY(check_csr(M));
  if (!val_out && M->nnz > 0) return TSPG_EINVAL;
  TSPG_CUDA(ctx, cudaSetDevice(ctx->device));
  cudaStream_t s = (cudaStream_t)stream;
  if (M->val_bits == 64)
    return M->rowptr_bits == 32 ? mcl_rows_impl<int32_t, double>(ctx, s, M, power, do_pow, val_out)
                                : mcl_rows_impl<int64_t, double>(ctx, s, M, power, do_pow, val_out);
  return M->rowptr_bits == 32 ? mcl_rows_impl<int32_t, float>(ctx, s, M, power, do_pow, val_out)
                              : mcl_rows_impl<int64_t, float>(ctx, s, M, power, do_pow, val_out);
}

extern "C" int tspg_mcl_normalize(tspg_ctx *ctx, void *stream, const tspg_csr *M, void *val_out) {
  return mcl_rows(ctx, stream, M, 1.0, 0, val_out);
}

extern "C" int tspg_mcl_inflate(tspg_ctx *ctx, void *stream, const tspg_csr *M, double power,
                                void *val_out) {
  return mcl_rows(ctx, stream, M, power, 1, val_out);
}

extern "C" int tspg_mcl_prune(tspg_ctx *ctx, void *stream, const tspg_csr *M, double tol,
                              tspg_csr_out *out) {
  if (!ctx || !out) return TSPG_EINVAL;
  TSPG_TRY(check_csr(M));
  if (!out->rowptr || out->nrows != M->nrows || out->ncols != M->ncols ||
      out->val_bits != M->val_bits || (out->rowptr_bits != 32 && out->rowptr_bits != 64))
    return TSPG_EINVAL;
  TSPG_CUDA(ctx, cudaSetDevice(ctx->device));
  cudaStream_t s = (cudaStream_t)stream;
  if (M->val_bits == 64)
    return M->rowptr_bits == 32 ? prune_impl<int32_t, double>(ctx, s, M, tol, out)
                                : prune_impl<int64_t, double>(ctx, s, M, tol, out);
  return M->rowptr_bits == 32 ? prune_impl<int32_t, float>(ctx, s, M, tol, out)
                              : prune_impl<int64_t, float>(ctx, s, M, tol, out);
}
