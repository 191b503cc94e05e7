// Test-only: the integer-pipe sums of fp64int.cuh against the additions they
// stand for, bit for bit, over seeded operands that fall like a stencil's
// (values of one size, values that cancel, values near zero and zeros beside
// large ones, short significands that make ties) and over a table of edge cases.
// Compiled by nvcc (kernels) or by the host compiler with the intrinsics
// spelled out below.  Built and run by tests/test_fxp.py.
#include <cstdint>
#include <cstring>

#ifndef __CUDACC__
#define __device__
#define __forceinline__ inline
#include <algorithm>
using std::max;
using std::min;
static long long bits_(double a) {
  long long u;
  memcpy(&u, &a, 8);
  return u;
}
static int __double2hiint(double a) { return (int)(bits_(a) >> 32); }
static int __double2loint(double a) { return (int)bits_(a); }
static double __hiloint2double(int h, int l) {
  long long u = ((long long)h << 32) | (unsigned)l;
  double a;
  memcpy(&a, &u, 8);
  return a;
}
static long long __double_as_longlong(double a) { return bits_(a); }
static double __longlong_as_double(long long u) { return __hiloint2double((int)(u >> 32), (int)u); }
static int __clz(int x) { return x ? __builtin_clz((unsigned)x) : 32; }
static unsigned __funnelshift_r(unsigned lo, unsigned hi, unsigned s) {
  return (unsigned)((((unsigned long long)hi << 32) | lo) >> (s & 31));
}
static unsigned __funnelshift_l(unsigned lo, unsigned hi, unsigned s) {
  return (unsigned)(((((unsigned long long)hi << 32) | lo) << (s & 31)) >> 32);
}
static double __dadd_rn(double a, double b) { return a + b; }
static double __dsub_rn(double a, double b) { return a - b; }
static double __dmul_rn(double a, double b) { return a * b; }
#define FXP_HOST
#endif
#include "fp64int.cuh"

namespace {

__device__ inline unsigned long long splitmix(unsigned long long x) {
  x += 0x9E3779B97F4A7C15ull;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
  return x ^ (x >> 31);
}

// seven operands of case t
__device__ inline void draw(unsigned long long t, unsigned long long seed, double* a) {
  unsigned long long u = splitmix(seed ^ (t * 0xD1B54A32D192ED03ull));
  const int kind = (int)(u % 6);
  const int e0 = (int)((u >> 8) % 200) - 100;
  const int spread = kind == 0 ? 1 : (kind == 1 ? 8 : (kind == 2 ? 40 : (kind == 3 ? 3 : 12)));
  for (int i = 0; i < 7; i++) {
    u = splitmix(u);
    unsigned long long m = u & 0xFFFFFFFFFFFFFull;
    u = splitmix(u);
    if (kind >= 3) {  // short significands: ties and exact cancellations
      const int keep = (int)((u >> 3) % 53);
      m &= ~((1ull << keep) - 1ull);
      if (u & 4) m |= 1ull << keep;
    }
    const int e = e0 - (int)((u >> 16) % (unsigned)spread);
    a[i] = __longlong_as_double((long long)(((u >> 63) << 63) | ((unsigned long long)(e + 1023) << 52) |
                                            (m & 0xFFFFFFFFFFFFFull)));
    if (kind == 5 && i && (u >> 40) % 3 == 0) a[i] = -a[i - 1];
    if (kind == 4 && (u >> 40) % 4 == 0) a[i] = (u >> 50) & 1 ? 0.0 : -0.0;
    if (kind == 1 && i && (u >> 40) % 5 == 0)  // a neighbour's value, one unit in the last place away
      a[i] = -__longlong_as_double(__double_as_longlong(a[i - 1]) + (long long)((u >> 45) % 3) - 1);
  }
}

__device__ inline bool same(double x, double y) {
  return __double_as_longlong(x) == __double_as_longlong(y) || (x != x && y != y);
}
// 0 when sum<6>, sum<4>, sum<2>, lap6, triple and scaled have the operations' bits
__device__ inline int check(const double* a) {
  double s2 = __dadd_rn(a[0], a[1]), s = __dadd_rn(s2, a[2]);
  s = __dadd_rn(s, a[3]);
  const double s4 = s;
  s = __dadd_rn(s, a[4]);
  s = __dadd_rn(s, a[5]);
  const double l = __dsub_rn(s, __dmul_rn(6.0, a[6]));
  const double v[6] = {a[0], a[1], a[2], a[3], a[4], a[5]}, v4[4] = {a[0], a[1], a[2], a[3]}, v2[2] = {a[0], a[1]};
  return !same(bsamg::fxp::sum<6>(v), s) + 2 * !same(bsamg::fxp::sum<4>(v4), s4) +
         4 * !same(bsamg::fxp::sum<2>(v2), s2) + 8 * !same(bsamg::fxp::lap6(v, a[6]), l) +
         16 * !same(bsamg::fxp::triple(a[6]), __dmul_rn(3.0, a[6])) +
         32 * !(same(bsamg::fxp::scaled<1>(a[6]), __dmul_rn(a[6], 2.0)) &&
                same(bsamg::fxp::scaled<-2>(a[5]), __dmul_rn(a[5], 0.25)) &&
                same(bsamg::fxp::scaled<-6>(a[6]), __dmul_rn(a[6], 1.0 / 64.0)));
}

}  // namespace

#ifdef FXP_HOST
extern "C" int fxp_random(unsigned long long n, unsigned long long seed, unsigned long long* bad, double* first) {
  *bad = 0;
  for (unsigned long long t = 0; t < n; t++) {
    double a[7];
    draw(t, seed, a);
    if (check(a) && (*bad)++ == 0) memcpy(first, a, sizeof(a));
  }
  return 0;
}
extern "C" int fxp_rows(const double* rows, int n, unsigned long long* bad, double* first) {
  *bad = 0;
  for (int t = 0; t < n; t++)
    if (check(rows + 7 * t) && (*bad)++ == 0) memcpy(first, rows + 7 * t, 56);
  return 0;
}
#else
namespace {
__global__ void k_random(unsigned long long n, unsigned long long seed, unsigned long long* bad, double* first) {
  for (unsigned long long t = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; t < n;
       t += (unsigned long long)gridDim.x * blockDim.x) {
    double a[7];
    draw(t, seed, a);
    if (check(a) && atomicAdd(bad, 1ull) == 0)
      for (int i = 0; i < 7; i++) first[i] = a[i];
  }
}
__global__ void k_rows(const double* rows, int n, unsigned long long* bad, double* first) {
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x)
    if (check(rows + 7 * t) && atomicAdd(bad, 1ull) == 0)
      for (int i = 0; i < 7; i++) first[i] = rows[7 * t + i];
}
struct Out {
  unsigned long long bad;
  double first[7];
};
int finish(Out* d, unsigned long long* bad, double* first) {
  Out h;
  cudaError_t e = cudaMemcpy(&h, d, sizeof(h), cudaMemcpyDeviceToHost);
  cudaFree(d);
  *bad = h.bad;
  memcpy(first, h.first, sizeof(h.first));
  return e == cudaSuccess ? 0 : 1;
}
}  // namespace
extern "C" int fxp_random(unsigned long long n, unsigned long long seed, unsigned long long* bad, double* first) {
  Out* d = nullptr;
  if (cudaMalloc(&d, sizeof(Out)) != cudaSuccess || cudaMemset(d, 0, sizeof(Out)) != cudaSuccess) return 1;
  k_random<<<152 * 4, 256>>>(n, seed, &d->bad, d->first);
  return finish(d, bad, first);
}
extern "C" int fxp_rows(const double* rows, int n, unsigned long long* bad, double* first) {
  Out* d = nullptr;
  double* r = nullptr;
  if (cudaMalloc(&d, sizeof(Out)) != cudaSuccess || cudaMemset(d, 0, sizeof(Out)) != cudaSuccess) return 1;
  if (cudaMalloc(&r, 56 * (size_t)n) != cudaSuccess) return 1;
  cudaMemcpy(r, rows, 56 * (size_t)n, cudaMemcpyHostToDevice);
  k_rows<<<152, 256>>>(r, n, &d->bad, d->first);
  const int rc = finish(d, bad, first);
  cudaFree(r);
  return rc;
}
#endif
