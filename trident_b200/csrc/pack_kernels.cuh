// pack_kernels.cuh — device kernels of the bitmask tile pack (masked segment
// counts and the copy pass), shared by tspg_pack and tspg_pack_noalloc.
#pragma once

#include <type_traits>

#include "internal.cuh"

namespace tspg {

// Masked segment lengths (select_ptrs' MaskedTransform, spacomm.cuh:539-553).
template <typename PT>
__global__ void k_pack_counts(const PT *ptr, int64_t len, const uint8_t *mask,
                              int32_t *cnt, uint32_t *ticket = nullptr) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (ticket && i == 0) *ticket = 0;  // of the scan to come
  if (i < len) {
    const bool keep = (mask[i >> 3] >> (i & 7)) & 1;
    cnt[i] = keep ? int32_t(int64_t(ptr[i + 1]) - int64_t(ptr[i])) : 0;
  }
}

// Copy pass, over the kept entries in output order: a warp takes runs of
// kPackRun of them (balanced however the entries cluster in segments).  Output
// entry o belongs to the last segment r with newp[r] <= o (the reference's
// locate_segment_by_pos, spacomm.cuh:714-725, on the packed offsets, in which
// masked segments are empty) and comes from ptr[r] + (o - newp[r]).  The
// pointer region starts at kept*(val+4) bytes rounded up to the pointer width
// (no padding for the reference's int32 pointers; at most 4 bytes for int64
// ones).  (Each thread walking 8 consecutive input entries behind a binary
// search of its own took 48 us for the 0.7M entries of an R-MAT tile.)
constexpr int kPackRun = 128;
template <typename PT, int VB>
__global__ void __launch_bounds__(256)
    k_pack_copy(const PT *ptr, int64_t len, const int32_t *idx, const void *val,
                const int64_t *newp, char *out, int64_t *kept_dev) {
  using V = typename std::conditional<VB == 8, unsigned long long, unsigned>::type;
  constexpr int U = kPackRun / 32;
  const int64_t kept = newp[len];
  V *oval = (V *)out;
  int32_t *oidx = (int32_t *)(out + kept * VB);
  const V *ival = (const V *)val;
  const int lane = threadIdx.x & 31;
  const int64_t t = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  const int64_t stride = int64_t(gridDim.x) * blockDim.x;
  // entries (an empty pointer array, len == 0, may be null and holds none)
  for (int64_t o0 = (t >> 5) * kPackRun; o0 < kept; o0 += (stride >> 5) * kPackRun) {
    int64_t r = first_row(newp, len, 0, o0, lane);
    int64_t src[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t o = o0 + u * 32 + lane;
      src[u] = -1;
      if (o0 + u * 32 < kept) {  // uniform
        const int64_t mine = window_row(newp, len, 0, r, o, lane);
        if (o < kept) src[u] = int64_t(ptr[mine]) + (o - newp[mine]);
      }
    }
    V v[U];
    int32_t c[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (src[u] >= 0) {
        v[u] = ival[src[u]];
        c[u] = idx[src[u]];
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t o = o0 + u * 32 + lane;
      if (src[u] >= 0) {
        oval[o] = v[u];
        oidx[o] = c[u];
      }
    }
  }
  // pointer array of the packed tile
  PT *optr = (PT *)(out + ((kept * (VB + 4) + int64_t(sizeof(PT)) - 1) &
                           ~(int64_t(sizeof(PT)) - 1)));
  for (int64_t i = t; i <= len; i += stride) optr[i] = PT(newp[i]);
  if (t == 0 && kept_dev) *kept_dev = kept;
}

}  // namespace tspg
