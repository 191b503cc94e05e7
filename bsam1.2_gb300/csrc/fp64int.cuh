// IEEE double sums and quotients on the integer pipe.
//
// GB300 issues one FP64 warp instruction per scheduler every 77 cycles (64
// when a warp is alone on its SM), against about one integer instruction a
// cycle, so a kernel bound by the FP64 unit leaves the integer pipe idle.
// The functions here evaluate a fixed sequence of round-to-nearest-even
// additions in fixed point and return the bits the additions return: the
// operands are aligned to the largest exponent in a frame of 96 bits, which
// holds all their bits, each partial sum is rounded to 53 significant bits
// where it stands, and the last one is packed.  Where an operand is
// subnormal, 2^-32 of the largest one, huge, infinite or NaN, or the result
// cancels to less than 2^-26 of the largest operand, the additions are done
// as additions.
//
// Measured (GB300), a 3D CH sweep of 256^3, a colour: 38 FP64 instructions a
// cell, 612 us; 27 with the sums and about 500 integer ones, 440 us; 16 with
// the two quotients, 312 us (each sum's last term is an FP64 addition again,
// see sum6: 17).  The residual norm: 15 instead of 32.
#pragma once
#ifndef FXP_CPU  // a test compiles this file for the host, with the intrinsics it spells out
#include <cuda_runtime.h>
#endif

namespace bsamg {
namespace fxp {

// The operations themselves, where the frame does not serve: called, not
// inlined, because a short block of FP64 instructions under a condition is
// issued predicated off on the common path too, and costs as much there.
#ifdef FXP_CPU
#define FXP_CALL static inline
#else
#define FXP_CALL static __device__ __noinline__
#endif
FXP_CALL double plain_add(double a, double b) { return __dadd_rn(a, b); }
FXP_CALL double plain_mul(double a, double b) { return __dmul_rn(a, b); }
FXP_CALL double plain_sum6(double a, double b, double c, double d, double e, double f) {
  return __dadd_rn(__dadd_rn(__dadd_rn(__dadd_rn(__dadd_rn(a, b), c), d), e), f);
}

// a partial sum h:l:x, two's complement, in units of 2^(E - 1023 - 84 - F)
struct Acc {
  int h;
  unsigned l, x;
};

__device__ __forceinline__ int exponent(double a) { return (__double2hiint(a) >> 20) & 0x7ff; }

// What decides whether the frame serves: the largest high word without its
// sign, and the smallest magnitude of a nonzero operand (its high word, the
// low one as a last bit, less one so that zeros come out largest)
struct Range {
  int top;
  unsigned low;
};
__device__ __forceinline__ void widen(Range& R, double a) {
  const int hi = __double2hiint(a) & 0x7fffffff;
  R.top = max(R.top, hi);
  R.low = min(R.low, ((unsigned)hi | min((unsigned)__double2loint(a), 1u)) - 1u);
}
// (a subnormal operand lies 2^-32 below any E >= 130)
__device__ __forceinline__ bool serves(const Range& R) {
  const int E = R.top >> 20;
  return E - (int)(R.low >> 20) < 32 && (unsigned)(E - 130) < 1800u;
}

// add h:l:x, negated when sign is -1
__device__ __forceinline__ void add96(Acc& A, unsigned h, unsigned l, unsigned x, int sign) {
#ifdef __CUDA_ARCH__
  unsigned t;  // its addition carries out when sign is -1
  asm("add.cc.u32 %3, %7, %7;\n\taddc.cc.u32 %0, %0, %4;\n\taddc.cc.u32 %1, %1, %5;\n\taddc.u32 %2, %2, %6;"
      : "+r"(A.x), "+r"(A.l), "+r"(A.h), "=r"(t)
      : "r"(x ^ (unsigned)sign), "r"(l ^ (unsigned)sign), "r"(h ^ (unsigned)sign), "r"(sign));
#else
  __int128 v = ((__int128)h << 64) | ((__int128)l << 32) | x;
  __int128 s = ((__int128)A.h << 64) | ((__int128)A.l << 32) | A.x;
  s += sign ? -v : v;
  A.h = (int)(s >> 64);
  A.l = (unsigned)(s >> 32);
  A.x = (unsigned)s;
#endif
}
// add a; top: the largest exponent E and ones below it, so that the
// subtraction of a high word borrows nothing from its exponent's place
template <int F>
__device__ __forceinline__ void add_value(Acc& A, double a, int top) {
  const int hi = __double2hiint(a);
  const unsigned lo = (unsigned)__double2loint(a);
  const unsigned d = (unsigned)(top - hi) >> 20;  // E - e in the low five bits, which are all a funnel shift takes
  const unsigned m = ((unsigned)hi & 0xfffffu) | (unsigned)min(hi & 0x7fffffff, 0x100000);  // a zero adds nothing
  const unsigned h = __funnelshift_l(lo, m, F), l = lo << F;
  add96(A, __funnelshift_r(h, 0u, d), __funnelshift_r(l, h, d), __funnelshift_r(0u, l, d), hi >> 31);
}
// round the partial sum to 53 significant bits, ties to even
__device__ __forceinline__ void round53(Acc& A) {
  const int sh = 11 - __clz(A.h ^ (A.h >> 31));  // bits of h:l below the 53rd
  const bool low = A.x != 0 && sh < 2;
  if (low) {  // a sum that cancelled: the 53rd bit is at 32 + sh of l:x
    const int neg = A.h >> 31;
    const int r = max(A.h != neg ? 32 + sh : 11 - __clz((int)(A.l ^ (unsigned)neg)), 0);
    unsigned long long u = ((unsigned long long)A.l << 32) | A.x;
    const unsigned long long mask = (1ull << r) - 1ull, half = mask >> 1;
    const unsigned long long v = u + half + ((u >> r) & mask & 1ull);
    A.h += v < u;
    A.l = (unsigned)((v & ~mask) >> 32);
    A.x = (unsigned)(v & ~mask);
  }
  // else x only says that the sum lies above l, which l's last bit says as
  // well when the rounding is at least two bits above it
  const int s = low ? 0 : max(sh, 0);
  const unsigned l = low ? A.l : A.l | min(A.x, 1u);
  A.x = low ? A.x : 0u;
  const unsigned mask = (1u << s) - 1u;
  const unsigned v = l + (mask >> 1) + ((l >> s) & mask & 1u);
  A.h += v < l;
  A.l = v & ~mask;
}
// the double of a rounded partial sum; ok: it is not smaller than 2^64 units
template <int F>
__device__ __forceinline__ double pack(const Acc& A, int E, bool& ok) {
  Acc u{0, 0u, 0u};
  const int neg = A.h >> 31;
  add96(u, (unsigned)A.h, A.l, A.x, neg);
  const int c = __clz(u.h) & 31;
  ok = u.h != 0;
  const unsigned th = __funnelshift_l(u.l, (unsigned)u.h, c), tl = __funnelshift_l(u.x, u.l, c);
  const unsigned mh = (th >> 11) & 0xfffffu, ml = __funnelshift_r(tl, th, 11);
  return __hiloint2double((int)(mh | ((unsigned)(E + 11 - F - c) << 20) | ((unsigned)neg & 0x80000000u)), (int)ml);
}

// RN(... RN(RN(a[0] + a[1]) + a[2]) ... + a[N-1]), N <= 6
// (seven bits above a significand and the sign leave room for six of them)
template <int N>
__device__ __forceinline__ double sum(const double (&a)[N]) {
  Range R{0, 0xffffffffu};
#pragma unroll
  for (int i = 0; i < N; i++) widen(R, a[i]);
  const int E = R.top >> 20, top = R.top | 0xfffff;
  Acc A{0, 0u, 0u};
#pragma unroll
  for (int i = 0; i < N; i++) {
    add_value<7>(A, a[i], top);
    if (i) round53(A);
  }
  bool ok;
  double r = pack<7>(A, E, ok);
  if (!(ok && serves(R))) {
    if constexpr (N == 6) {
      r = plain_sum6(a[0], a[1], a[2], a[3], a[4], a[5]);
    } else {
      r = a[0];
#pragma unroll
      for (int i = 1; i < N; i++) r = plain_add(r, a[i]);
    }
  }
  return r;
}

// RN(.. + a[5]) with the first five terms on the integer pipe: an addition is
// about 40 instructions there, as long as the FP64 unit takes for one, and
// with one or two of them left to it both pipes are busy alike (256^3 sweep:
// six terms 344 us, five 321, four 329)
__device__ __forceinline__ double sum6(const double (&a)[6]) {
  return __dadd_rn(sum<5>({a[0], a[1], a[2], a[3], a[4]}), a[5]);
}

// RN(3 x): a significand times three has 54 or 55 bits
__device__ __forceinline__ double triple(double x) {
  const int hi = __double2hiint(x), e = (hi >> 20) & 0x7ff;
  const unsigned long long m =
      ((unsigned long long)(((unsigned)hi & 0xfffffu) | 0x100000u) << 32) | (unsigned)__double2loint(x);
  unsigned long long m3 = m + (m << 1);
  const int r = 1 + ((int)(m3 >> 54) & 1);
  m3 += ((1u << r) >> 1) - 1u + (((unsigned)m3 >> r) & 1u);
  m3 >>= r;  // its leading bit, or a carry into the next power of two, adds to the exponent
  double y = __hiloint2double((hi & (int)0x80000000u) | ((int)(m3 >> 32) + ((e + r - 1) << 20)), (int)m3);
  if ((unsigned)(e - 1) >= 2040u) y = plain_mul(3.0, x);
  return y;
}
// x 2^k, |k| < 8
template <int K>
__device__ __forceinline__ double scaled(double x) {
  const int hi = __double2hiint(x), e = (hi >> 20) & 0x7ff;
  double y = __hiloint2double(hi + K * (1 << 20), __double2loint(x));
  if ((unsigned)(e - 8) >= 2030u) y = plain_mul(x, K < 0 ? 1.0 / (1 << (K < 0 ? -K : 0)) : 1.0 * (1 << (K > 0 ? K : 0)));
  return y;
}

// RN(sum(a) - RN(6 c)): the undivided Laplacian of the six neighbours (the
// norm of 160x96x128 with the centre in the frame too 88 us, so 80, with five
// terms 83; 3 c on the integer pipe as well made the norm of 250^3 532 -> 568)
__device__ __forceinline__ double lap6(const double (&a)[6], double c) {
  return __dadd_rn(sum<6>(a), -__dmul_rn(6.0, c));
}

// ---- quotients ----
//
// RN(a / b) needs seven FP64 instructions for a correctly rounded reciprocal
// and three for each quotient; on the integer pipe it is a reciprocal of 60
// bits (35 instructions) and, for each quotient, a product, a remainder and
// one comparison (40).  Two quotients of one divisor share the reciprocal.
//
// The significand of b as D in [2^63, 2^64); x = 2^63 / D in (0.5, 1].  A
// single-precision reciprocal of D's leading 24 bits is x to 2^-21.7, a
// Newton step x (2 - x / x_true) to 2^-42.9 and another to 2^-59.8, where
// the steps' truncations are kept on one side: the result never exceeds x,
// so that neither does the quotient T with ten bits below its last place,
// and T, rounded, is the correctly rounded quotient or the value below it.
// The remainder, exact modulo 2^64, tells which; there are no ties.
FXP_CALL double plain_div(double a, double b) { return a / b; }

#ifdef FXP_CPU
#ifndef FXP_SEED_ULPS
#define FXP_SEED_ULPS 0
#endif
static inline unsigned seed_bits(unsigned d) {  // the device's approximation is within one unit of this
  float f, r;
  memcpy(&f, &d, 4);
  r = 1.0f / f;
  unsigned u;
  memcpy(&u, &r, 4);
  return u + FXP_SEED_ULPS;
}
#else
__device__ __forceinline__ unsigned seed_bits(unsigned d) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float(d)));
  return __float_as_uint(r);
}
#endif

// a divisor: its significand m in [2^52, 2^53), its exponent and y = x 2^64,
// at most 10 units low
struct Divisor {
  unsigned long long m, y;
  int e;
};
__device__ __forceinline__ Divisor divisor(double b) {
  Divisor r;
  const unsigned hi = (unsigned)__double2hiint(b), lo = (unsigned)__double2loint(b);
  r.e = (int)(hi >> 20);  // b > 0
  const unsigned mh = (hi & 0xfffffu) | 0x100000u;
  r.m = ((unsigned long long)mh << 32) | lo;
  const unsigned dh = __funnelshift_l(lo, mh, 11), dl = lo << 11;
  // y0 = x 2^32: the seed's 24 bits (a seed of 1 counts as the value below it)
  const unsigned s = seed_bits(0x3f800000u | ((dh >> 8) & 0x7fffffu));
  const unsigned y0 = (min((int)s, 0x3f7fffff) << 8) | 0x80000000u;
  // 1 - x^-1 y0 in units of 2^-52, below 2^31
  const unsigned long long p = (unsigned long long)dh * y0 + (((unsigned long long)dl * y0) >> 32);
  const int e1 = (int)((long long)(0x8000000000000000ull - p) >> 11);
  const unsigned long long y1 = ((unsigned long long)y0 << 32) + (unsigned long long)(((long long)e1 * (int)(y0 >> 1)) >> 19);
  // 1 - x^-1 y1 in units of 2^-63, below 2^21: its low 32 bits are all of it
  const unsigned yh = (unsigned)(y1 >> 32), yl = (unsigned)y1;
  const unsigned long long c1 = (unsigned long long)dl * yh, c2 = (unsigned long long)dh * yl;
  const unsigned long long mid = (c1 & 0xffffffffull) + (c2 & 0xffffffffull);
  const unsigned low = dh * yh + (unsigned)(c1 >> 32) + (unsigned)(c2 >> 32) + (unsigned)(mid >> 32);
  const int e2 = -(int)low - 4;  // four units to stay below x, whatever was cut off
  r.y = y1 + (unsigned long long)(((long long)e2 * (int)(yh >> 1)) >> 30);
  return r;
}
// 1 <= b < 2^400 and 2^-400 <= |a| < 2^400: quotients in the normal range
__device__ __forceinline__ bool divides(double b) { return ((unsigned)__double2hiint(b) >> 20) - 1023u < 400u; }
__device__ __forceinline__ bool divisible(double a) { return (unsigned)(exponent(a) - (1023 - 400)) <= 799u; }
__device__ __forceinline__ double quotient(double a, const Divisor& b) {
  const unsigned hi = (unsigned)__double2hiint(a), lo = (unsigned)__double2loint(a);
  unsigned long long A = ((unsigned long long)((hi & 0xfffffu) | 0x100000u) << 32) | lo;
  const int half = A < b.m;  // a quotient of significands in [1, 2)
  A <<= half;
#ifdef FXP_CPU
  const unsigned long long T = (unsigned long long)(((unsigned __int128)(A << 10) * b.y) >> 64);
#else
  const unsigned long long T = __umul64hi(A << 10, b.y);
#endif
  unsigned long long q = (T + 512u) >> 10;
  const long long rem = (long long)((A << 52) - q * b.m);
  q += 2 * rem > (long long)b.m;
  const int e = (int)((hi >> 20) & 0x7ff) - b.e + 1023 - half;
  return __hiloint2double((int)(((hi & 0x80000000u) | ((unsigned)(e - 1) << 20)) + (unsigned)(q >> 32)), (int)q);
}
// RN(a / b)
__device__ __forceinline__ double quot(double a, double b) {
  double q = quotient(a, divisor(b));
  if (!(divides(b) && divisible(a))) q = plain_div(a, b);
  return q;
}
// RN(a0 / b), RN(a1 / b)
__device__ __forceinline__ void quot2(double a0, double a1, double b, double& q0, double& q1) {
  const Divisor d = divisor(b);
  q0 = quotient(a0, d);
  q1 = quotient(a1, d);
  if (!(divides(b) && divisible(a0) && divisible(a1))) {
    q0 = plain_div(a0, b);
    q1 = plain_div(a1, b);
  }
}

}  // namespace fxp
}  // namespace bsamg
