// Test-only: the integer-pipe quotients of fp64int.cuh against `/`, bit for
// bit, on the host (the intrinsics spelled out): seeded operands over the
// fast form's range, quotients next to a rounding boundary, and a table of
// edge cases.  FXP_SEED_ULPS moves the single-precision seed as far as the
// device's approximate reciprocal may be off.  Built by tests/test_fxq_cpu.py.
#include <cstdint>
#include <cstring>
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
static double of_bits(unsigned long long u) {
  double a;
  memcpy(&a, &u, 8);
  return a;
}
static int __clz(int x) { return x ? __builtin_clz((unsigned)x) : 32; }
static unsigned __funnelshift_r(unsigned lo, unsigned hi, unsigned s) {
  return (unsigned)((((unsigned long long)hi << 32) | lo) >> (s & 31));
}
static unsigned __funnelshift_l(unsigned lo, unsigned hi, unsigned s) {
  return (unsigned)(((((unsigned long long)hi << 32) | lo) << (s & 31)) >> 32);
}
static double __dadd_rn(double a, double b) { return a + b; }
static double __dmul_rn(double a, double b) { return a * b; }
#include "fp64int.cuh"

static unsigned long long splitmix(unsigned long long x) {
  x += 0x9E3779B97F4A7C15ull;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
  return x ^ (x >> 31);
}
static bool same(double x, double y) { return bits_(x) == bits_(y) || (x != x && y != y); }
static bool check(double a, double a1, double b) {
  double q0, q1;
  bsamg::fxp::quot2(a, a1, b, q0, q1);
  return same(q0, a / b) && same(q1, a1 / b) && same(bsamg::fxp::quot(a, b), a / b);
}
extern "C" unsigned long long fxq_random(unsigned long long n, unsigned long long seed, double* first) {
  unsigned long long bad = 0;
  for (unsigned long long t = 0; t < n; t++) {
    unsigned long long u = splitmix(seed ^ (t * 0xD1B54A32D192ED03ull)), v = splitmix(u), w = splitmix(v);
    const int kind = (int)(w % 4);
    unsigned long long mb = u & 0xFFFFFFFFFFFFFull, ma = v & 0xFFFFFFFFFFFFFull;
    if (kind == 1) mb &= ~0ull << (w / 4 % 53);                                       // short divisors
    if (kind == 2) mb = (w & 4) ? 0xFFFFFFFFFFFFFull - (u % 64) : u % 64;             // next to a power of two
    const double b = of_bits(((unsigned long long)(1023 + (w >> 8) % (kind ? 30 : 399)) << 52) | mb);
    double a = of_bits(((w >> 63) << 63) | ((unsigned long long)(1023 - 399 + (w >> 20) % 798) << 52) | ma);
    if (kind == 3) {  // a quotient next to the middle of two values: b (q + half a unit), rounded
      const double q = of_bits((1023ull << 52) | ma);
      a = (double)((long double)b * ((long double)q + 0x1p-53L));
    }
    if (!check(a, -of_bits(bits_(a) ^ (u >> 40 & 7)), b) && bad++ == 0) first[0] = a, first[1] = b;
  }
  return bad;
}
extern "C" unsigned long long fxq_rows(const double* rows, int n, double* first) {
  unsigned long long bad = 0;
  for (int t = 0; t < n; t++)
    if (!check(rows[3 * t], rows[3 * t + 1], rows[3 * t + 2]) && bad++ == 0) memcpy(first, rows + 3 * t, 24);
  return bad;
}
