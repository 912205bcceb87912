// C++ GPU test: a process that resets its device and goes on with a new
// context.  The kernels' shared-memory limits are gone with the old one, so a
// product and a transpose must raise them again.
#include <cuda_runtime.h>

#include <cstdio>
#include <vector>

#include "tspg.h"

static void *alloc(void *, size_t bytes, void *) {
  void *p = nullptr;
  return cudaMalloc(&p, bytes ? bytes : 1) == cudaSuccess ? p : nullptr;
}

template <typename T>
static T *up(const std::vector<T> &v) {
  T *p = (T *)alloc(nullptr, v.size() * sizeof(T), nullptr);
  cudaMemcpy(p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice);
  return p;
}

static bool once() {
  const int n = 300;
  std::vector<int64_t> rp(n + 1);
  std::vector<int32_t> col;
  std::vector<double> val;
  for (int i = 0; i < n; ++i) {
    for (int k = 0; k < 5; ++k) col.push_back(i / 5 * 5 + k), val.push_back(1.0);
    rp[i + 1] = int64_t(col.size());
  }
  tspg_ctx *ctx = nullptr;
  if (tspg_ctx_create(0, 0, &ctx) != TSPG_OK) return false;
  tspg_csr A{n, n, int64_t(col.size()), up(rp), 64, 64, up(col), up(val)};
  bool ok = true;
  for (int k = 0; k < 2; ++k) {
    tspg_csr_out C{};
    C.nrows = C.ncols = n;
    C.rowptr = alloc(nullptr, (n + 1) * 8, nullptr);
    C.rowptr_bits = C.val_bits = 64;
    C.alloc = alloc;
    const int st = k == 0 ? tspg_spgemm(ctx, nullptr, &A, &A, &C, 0) : tspg_transpose(ctx, nullptr, &A, &C);
    ok = ok && st == TSPG_OK && cudaDeviceSynchronize() == cudaSuccess && C.nnz == 5 * n;
    std::vector<double> v(5 * n);
    if (ok) cudaMemcpy(v.data(), C.val, v.size() * 8, cudaMemcpyDeviceToHost);
    for (double x : v) ok = ok && x == (k == 0 ? 5.0 : 1.0);
  }
  return tspg_ctx_destroy(ctx) == TSPG_OK && ok;
}

int main() {
  bool ok = true;
  for (int k = 0; k < 3; ++k) {
    ok = once() && ok;
    ok = cudaDeviceReset() == cudaSuccess && ok;
  }
  std::printf(ok ? "ALL OK\n" : "FAIL\n");
  return ok ? 0 : 1;
}
