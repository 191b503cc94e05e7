// Test-only: sum<5> and sum6 of fp64int.cuh, the forms the 3D sweeps call,
// against the additions they stand for, over the operands of fxp_check.cu.
// Built and run by tests/test_fxp_sum5.py.
#define check check_others
#include "fxp_check.cu"
#undef check

namespace {

// 0 when both have the additions' bits
__device__ inline int check5(const double* a) {
  double s5 = __dadd_rn(a[0], a[1]);
  for (int i = 2; i < 5; i++) s5 = __dadd_rn(s5, a[i]);
  const double v5[5] = {a[0], a[1], a[2], a[3], a[4]}, v6[6] = {a[0], a[1], a[2], a[3], a[4], a[5]};
  return !same(bsamg::fxp::sum<5>(v5), s5) + 2 * !same(bsamg::fxp::sum6(v6), __dadd_rn(s5, a[5]));
}

}  // namespace

#ifdef FXP_HOST
extern "C" int fxp_random5(unsigned long long n, unsigned long long seed, unsigned long long* bad, double* first) {
  *bad = 0;
  for (unsigned long long t = 0; t < n; t++) {
    double a[7];
    draw(t, seed, a);
    if (check5(a) && (*bad)++ == 0) memcpy(first, a, sizeof(a));
  }
  return 0;
}
extern "C" int fxp_rows5(const double* rows, int n, unsigned long long* bad, double* first) {
  *bad = 0;
  for (int t = 0; t < n; t++)
    if (check5(rows + 7 * t) && (*bad)++ == 0) memcpy(first, rows + 7 * t, 56);
  return 0;
}
#else
namespace {
// case t of n: row t, or drawn from the seed when there are no rows
__global__ void k_check5(const double* rows, unsigned long long n, unsigned long long seed, Out* out) {
  for (unsigned long long t = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; t < n;
       t += (unsigned long long)gridDim.x * blockDim.x) {
    double a[7];
    if (rows)
      for (int i = 0; i < 7; i++) a[i] = rows[7 * t + i];
    else
      draw(t, seed, a);
    if (check5(a) && atomicAdd(&out->bad, 1ull) == 0)
      for (int i = 0; i < 7; i++) out->first[i] = a[i];
  }
}
int run5(const double* rows, unsigned long long n, unsigned long long seed, unsigned long long* bad, double* first) {
  Out* d = nullptr;
  double* r = nullptr;
  if (cudaMalloc(&d, sizeof(Out)) != cudaSuccess || cudaMemset(d, 0, sizeof(Out)) != cudaSuccess) return 1;
  if (rows && (cudaMalloc(&r, 56 * n) != cudaSuccess || cudaMemcpy(r, rows, 56 * n, cudaMemcpyHostToDevice) != cudaSuccess))
    return 1;
  k_check5<<<152 * 4, 256>>>(r, n, seed, d);
  const int rc = finish(d, bad, first);
  cudaFree(r);
  return rc;
}
}  // namespace
extern "C" int fxp_random5(unsigned long long n, unsigned long long seed, unsigned long long* bad, double* first) {
  return run5(nullptr, n, seed, bad, first);
}
extern "C" int fxp_rows5(const double* rows, int n, unsigned long long* bad, double* first) {
  return run5(rows, (unsigned long long)n, 0, bad, first);
}
#endif
