// Mixed-precision MultigridIterations on periodic boxes.
//
// Applies when every level of the hierarchy is one fully periodic patch with
// even extents that covers its parent (a uniform periodic grid and its
// below-root levels, RootInit/InitSeed, bsamroutines.f90:226-510).  The
// algorithm is the one of mixed.cu -- an FP32 FAS V-cycle on the correction
// equation M(e) = N(qbar + e) - N(qbar) = g inside an outer loop that updates
// qbar and confirms convergence on the true residual f - N(qbar) -- with a
// data layout and precision split chosen for GB300:
//
//  * No ghost cells and no work lists.  Neighbours wrap around the box, and
//    every kernel derives its cell from a 3D grid, so a thread's first loads
//    are its data (no dependent table lookups).
//  * Colour-split FP32 arrays (BoxLev).  A red half-sweep reads whole
//    sectors of black values and writes whole sectors of red ones, instead
//    of touching every sector of an interleaved array for half its bytes.
//  * The FP64 iterate is held for the whole solve as a pair of floats
//    (hi + lo, about 48 significant bits).  qbar += e is a TwoSum, and the
//    residual f - N(qbar) is evaluated in double-float arithmetic, all on the
//    FP32 pipe; GB300's FP64 rate is 1/64 of its FP32 rate.  The rounding
//    error of the double-float residual is about 2^-47 times the largest
//    term (|c0 ulap(mu)|, |phi^3| ~ 1-100 here), i.e. ~1e-12, four orders
//    below the 1e-8..1e-9 tolerances the residual is tested against.  FP64 is
//    used only to split q at the start (integer bit operations, exact) and
//    to write it back at the end (one FP64 add per value).
//  * The tracked residual update g <- g - M(e) and qbar += e are one pass,
//    and e is never cleared: the first two half-sweeps of a cycle on the
//    finest level treat the previous cycle's e as zero.
//
// Plugin: CH (CH/problem.f90), whose source is f = (phi_old, -phi_old)
// (Source2D/3D, :425-450, :672-695) and whose operator is
// N(q) = (phi - dt/h^2 ULap(mu), mu - phi^3 + eps^2/h^2 ULap(phi))
// (Operator2D/3D, :393-422, :638-669).
#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <cstddef>
#include <functional>
#include <memory>
#include <vector>

#include "box.h"
#include "kern_uni.cuh"
#include "launch.h"
#include "uni.h"

namespace bsamg {

namespace {

// colour of 0-based cell (x, y, z): parity of the 1-based i + j (+ k)
template <int DIM>
__device__ __forceinline__ int colour(int x, int y, int z) {
  return DIM == 3 ? (x + y + z + 1) & 1 : (x + y) & 1;
}

// A cell and its six neighbours as 32-bit indices into a colour-split array
// of one variable, the colour offset included: own = c*half + row*hh + x/2,
// the neighbours in the other colour's half.  A kernel forms one base
// pointer per array and variable (fp + offset + v*2*half), the same for all
// its threads, so that a load costs one address instruction.
template <int DIM>
struct Loc {
  int c;
  unsigned own, xm, xp, ym, yp, zm, zp;
  __device__ __forceinline__ Loc(const BoxLev& L, int x, int y, int z) {
    c = colour<DIM>(x, y, z);
    unsigned hh = (unsigned)L.hh, n1 = (unsigned)L.n[1], half = (unsigned)L.half;
    unsigned h = (unsigned)x >> 1, b = (unsigned)x & 1u;
    unsigned r = (unsigned)z * n1 + (unsigned)y;
    unsigned on = c ? 0u : half;  // start of the other colour
    own = (c ? half : 0u) + r * hh + h;
    unsigned row = on + r * hh;
    xm = row + (b ? h : (h ? h - 1 : hh - 1));
    xp = row + (b ? (h + 1 < hh ? h + 1 : 0u) : h);
    unsigned rz = r - (unsigned)y;  // z * n1
    ym = on + (rz + (y ? (unsigned)y - 1 : n1 - 1)) * hh + h;
    yp = on + (rz + ((unsigned)y + 1 < n1 ? (unsigned)y + 1 : 0u)) * hh + h;
    if (DIM == 3) {
      unsigned n2 = (unsigned)L.n[2];
      zm = on + ((z ? (unsigned)z - 1 : n2 - 1) * n1 + (unsigned)y) * hh + h;
      zp = on + (((unsigned)z + 1 < n2 ? (unsigned)z + 1 : 0u) * n1 + (unsigned)y) * hh + h;
    } else {
      zm = zp = 0;
    }
  }
};

template <int DIM, typename T = float>
__device__ __forceinline__ T nsum(const float* a, const Loc<DIM>& l) {
  T s = T(a[l.xm]) + T(a[l.xp]) + T(a[l.ym]) + T(a[l.yp]);
  if (DIM == 3) s += T(a[l.zm]) + T(a[l.zp]);
  return s;
}

// bases of variables 0 and 1 of a two-variable colour-split array
struct V2 {
  float* v0;
  float* v1;
};
__device__ __forceinline__ V2 var2(float* fp, long long off, long long half) {
  return {fp + off, fp + off + 2 * half};
}

// correction operator M(e) at a cell (see mixed.cu, mopn) whose variables'
// neighbours sum to s0 and s1
template <int DIM>
__device__ __forceinline__ void mop_cell(const BoxLev& L, float x, float y, float pb, float s0, float s1, float& m0,
                                         float& m1) {
  const float k = DIM == 2 ? 4.0f : 6.0f;
  m0 = x - L.c0 * (s1 - k * y);
  m1 = y - x * (3.0f * pb * (pb + x) + x * x) + L.c1 * (s0 - k * x);
}
template <int DIM>
__device__ __forceinline__ void mop(V2 E, const BoxLev& L, const Loc<DIM>& l, float pb, float& m0, float& m1) {
  mop_cell<DIM>(L, E.v0[l.own], E.v1[l.own], pb, nsum<DIM>(E.v0, l), nsum<DIM>(E.v1, l), m0, m1);
}

// the undivided Laplacian as a sum of neighbour differences: for a smooth
// correction each difference of two close values is exact (Sterbenz), so the
// rounding error is relative to the Laplacian, not to the values (the sum of
// neighbours minus k times the centre cancels and keeps ~1e-7 of |e|)
template <int DIM>
__device__ __forceinline__ float ndiff(const float* a, const Loc<DIM>& l, float c) {
  float s = ((a[l.xm] - c) + (a[l.xp] - c)) + ((a[l.ym] - c) + (a[l.yp] - c));
  if (DIM == 3) s += (a[l.zm] - c) + (a[l.zp] - c);
  return s;
}

// M(e) for the tracked residual g <- g - M(e): its rounding accumulates into
// the right-hand side of every later cycle (the smoother's and the coarse
// correction's only slow convergence down), so the Laplacians are evaluated
// in the difference form.  With c0 = dt/h^2 ~ 33 at 256^3 the summed form
// left a floor near 1e-5 |e| in g: from the 12th step on the last cycle of a
// step gained 5x instead of 12x, and later steps needed a sixth cycle.
template <int DIM>
__device__ __forceinline__ void mop_track(V2 E, const BoxLev& L, const Loc<DIM>& l, float pb, float& m0, float& m1) {
  float x = E.v0[l.own], y = E.v1[l.own];
  m0 = x - L.c0 * ndiff<DIM>(E.v1, l, y);
  m1 = y - x * (3.0f * pb * (pb + x) + x * x) + L.c1 * ndiff<DIM>(E.v0, l, x);
}

// ---------------------------------------------------------------------------
// double-float arithmetic (value = h + l, |l| <= ulp(h)/2 after
// normalisation): Dekker/Knuth error-free transformations

struct DF {
  float h, l;
};
__device__ __forceinline__ DF two_sum(float a, float b) {
  float s = a + b;
  float bb = s - a;
  return {s, (a - (s - bb)) + (b - bb)};
}
__device__ __forceinline__ DF fast_two_sum(float a, float b) {
  float s = a + b;
  return {s, b - (s - a)};
}
__device__ __forceinline__ DF df_add(DF x, DF y) {
  DF s = two_sum(x.h, y.h);
  return fast_two_sum(s.h, s.l + (x.l + y.l));
}
__device__ __forceinline__ DF df_neg(DF x) { return {-x.h, -x.l}; }
__device__ __forceinline__ DF df_mul(DF x, DF y) {
  float p = x.h * y.h;
  float e = fmaf(x.h, y.h, -p);
  e = fmaf(x.h, y.l, e);
  e = fmaf(x.l, y.h, e);
  return fast_two_sum(p, e);
}
// undivided Laplacian sum(neighbours) - k*centre of double-float values
template <int DIM>
__device__ __forceinline__ DF df_lap(const DF* nb, DF c) {
  float sh = nb[0].h, el = nb[0].l;
  for (int m = 1; m < 2 * DIM; m++) {
    DF t = two_sum(sh, nb[m].h);
    sh = t.h;
    el += t.l + nb[m].l;
  }
  const float k = DIM == 2 ? 4.0f : 6.0f;
  float p = k * c.h;
  float pe = fmaf(k, c.h, -p);  // k*c.h = p + pe exactly
  DF t = two_sum(sh, -p);
  el += t.l - pe - k * c.l;
  return fast_two_sum(t.h, el);
}

// Split a double into hi + lo floats with integer operations only (no FP64
// instructions).  hi keeps the leading 24 significant bits (truncated), lo
// the next 29 rounded to 24, so hi + lo carries 48 of the 53 bits.  Values
// whose magnitude is outside [2^-70, 2^120] (zero, denormals, infinities,
// NaN, extremes) take the conversion instructions instead.
__device__ __forceinline__ DF split64(double x) {
  unsigned long long b = (unsigned long long)__double_as_longlong(x);
  unsigned int top = (unsigned int)(b >> 32);
  int e = (int)((top >> 20) & 0x7FFu) - 1023;
  if (e >= -70 && e <= 120) {
    unsigned int s = top & 0x80000000u;
    float hi = __uint_as_float(s | ((unsigned int)(e + 127) << 23) | ((unsigned int)(b >> 29) & 0x7FFFFFu));
    float rf = __uint2float_rn((unsigned int)b & 0x1FFFFFFFu);
    float lo = rf * __uint_as_float((unsigned int)(e - 52 + 127) << 23);
    return {hi, s ? -lo : lo};
  }
  if ((b << 1) == 0) return {__uint_as_float(top & 0x80000000u), 0.0f};
  float hi = (float)x;
  return {hi, (float)(x - (double)hi)};
}
// float -> double by integer operations, every case of it: a conversion held
// back by a predicate still takes the FP64 unit's 64 cycles
__device__ __forceinline__ double f2d(float f) {
  const unsigned u = __float_as_uint(f), a = u & 0x7FFFFFFFu;
  unsigned hi = (a >> 3) + 0x38000000u, lo = u << 29;
  if (a - 0x00800000u >= 0x7F000000u) {  // zero, subnormal, infinite or NaN
    if (a >= 0x7F800000u) {
      hi = (a >> 3) + 0x70000000u;
    } else if (a == 0) {
      hi = 0;
    } else {  // the leading bit to the implicit place
      const int s = __clz(a) - 8;
      const unsigned m = a << s;
      hi = (m >> 3) + 0x38000000u - ((unsigned)s << 20);
      lo = m << 29;
    }
  }
  return __hiloint2double((int)(hi | (u & 0x80000000u)), (int)lo);
}

// deterministic per-CTA sums of two values -> partial[2*cta], [2*cta+1]:
// warp shuffles then one thread over the warp sums when the block is whole
// warps, else a shared-memory tree
__device__ __forceinline__ void cta_sum2(float s0, float s1, double* partial) {
  __shared__ float red[2][256];
  int t = threadIdx.y * blockDim.x + threadIdx.x;
  int nt = blockDim.x * blockDim.y;
  if ((nt & 31) == 0) {
    for (int o = 16; o > 0; o >>= 1) {
      s0 += __shfl_down_sync(0xffffffffu, s0, o);
      s1 += __shfl_down_sync(0xffffffffu, s1, o);
    }
    if ((t & 31) == 0) {
      red[0][t >> 5] = s0;
      red[1][t >> 5] = s1;
    }
    __syncthreads();
    if (t == 0)
      for (int w = 1; w < (nt >> 5); w++) {
        red[0][0] += red[0][w];
        red[1][0] += red[1][w];
      }
  } else {
    red[0][t] = s0;
    red[1][t] = s1;
    __syncthreads();
    for (int w = 128; w > 0; w >>= 1) {
      if (t < w && t + w < nt) {
        red[0][t] += red[0][t + w];
        red[1][t] += red[1][t + w];
      }
      __syncthreads();
    }
  }
  if (t == 0) {
    long long cta = ((long long)blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
    partial[2 * cta] = (double)red[0][0];
    partial[2 * cta + 1] = (double)red[1][0];
  }
}

// ---------------------------------------------------------------------------
// kernels.  Grid (x, y, z) = (position in a colour row or coarse x,
// y, z); blockDim.z = 1.

// The pointwise Newton update of one cell in FP32 (the 2x2 solve of
// RelaxGrid2D/3D in correction form), every rounding explicit so that each
// kernel that smooths computes the same bits whatever the compiler would
// contract:  a21 = -3 (pb + xv)^2 - tmp3,  b1 = g0 + c0 s1,
// b2 = g1 - c1 s0 - xv^2 (3 pb + 2 xv),  det = 1 - a12 a21,
// e0 = (b1 - a12 b2) / det,  e1 = (b2 - a21 b1) / det.
__device__ __forceinline__ void newton_cell(float c0, float c1, float tmp3, float a12, float pb, float xv, float s0,
                                            float s1, float g0, float g1, float& r0, float& r1) {
  const float w = __fadd_rn(pb, xv);
  const float a21 = __fmaf_rn(__fmul_rn(-3.0f, w), w, -tmp3);
  const float b1 = __fmaf_rn(c0, s1, g0);
  const float t = __fmaf_rn(3.0f, pb, __fmul_rn(2.0f, xv));
  const float b2 = __fmaf_rn(-__fmul_rn(xv, xv), t, __fmaf_rn(-c1, s0, g1));
  const float rdet = __frcp_rn(__fmaf_rn(-a12, a21, 1.0f));
  r0 = __fmul_rn(__fmaf_rn(-a12, b2, b1), rdet);
  r1 = __fmul_rn(__fmaf_rn(-a21, b1, b2), rdet);
}
__device__ __forceinline__ void newton_cell(const BoxLev& L, float pb, float xv, float s0, float s1, float g0,
                                            float g1, float& r0, float& r1) {
  newton_cell(L.c0, L.c1, L.tmp3, L.a12, pb, xv, s0, s1, g0, g1, r0, r1);
}

// One cell of a colour half-sweep of the correction smoother (RelaxGrid2D/3D
// in correction form, see mixed.cu k_mx_relax) in FP64 arithmetic with the
// FP64 coefficients (FP32 storage).  first = 1: e of both colours counts as
// zero (first half-sweep of a cycle); first = 2: the own colour's e counts as
// zero (second half-sweep).
template <int DIM>
__device__ __forceinline__ void relax64_at(float* __restrict__ fp, const BoxLev& L, int c, int first, int h, int y,
                                           int z) {
  V2 E = var2(fp, L.oe, L.half), G = var2(fp, L.og, L.half);
  int x = 2 * h + ((c + y + z + (DIM == 3 ? 1 : 0)) & 1);
  Loc<DIM> l(L, x, y, z);
  double pb = fp[L.opb + l.own], s0 = 0.0, s1 = 0.0, xv = 0.0;
  if (first != 1) {
    s0 = nsum<DIM, double>(E.v0, l);
    s1 = nsum<DIM, double>(E.v1, l);
    if (first == 0) xv = E.v0[l.own];
  }
  double w = pb + xv;
  double a21 = -3.0 * w * w - L.cd[2];
  double b1 = G.v0[l.own] + L.cd[0] * s1;
  double b2 = G.v1[l.own] - L.cd[1] * s0 - xv * xv * (3.0 * pb + 2.0 * xv);
  double rdet = 1.0 / (1.0 - L.cd[3] * a21);
  E.v0[l.own] = (float)((b1 - L.cd[3] * b2) * rdet);
  E.v1[l.own] = (float)((b2 - a21 * b1) * rdet);
}

// the FP64 smoother over a whole level (the coarsest level of a V-cycle
// that no small-level cycle covers): one cell of the colour per thread
template <int DIM>
__global__ void __launch_bounds__(256) k_bx_relax64(float* __restrict__ fp, BoxLev L, int c, int first) {
  after_previous();
  int h = blockIdx.x * blockDim.x + threadIdx.x;
  int y = blockIdx.y * blockDim.y + threadIdx.y;
  if (h < L.hh && y < L.n[1]) relax64_at<DIM>(fp, L, c, first, h, y, blockIdx.z);
}

// Full-grid sweep: each thread takes position h of rows R*yp .. R*yp+R-1
// (n1 is a multiple of R), loading all its cells' data before any is stored
// so that R times the loads are in flight per thread.
template <int DIM, int R = 2, int MINB = 8>
__global__ void __launch_bounds__(256, MINB) k_bx_relax(float* __restrict__ fp, BoxLev L, int c, int first) {
  after_previous();
  int h = blockIdx.x * blockDim.x + threadIdx.x;
  int yp = blockIdx.y * blockDim.y + threadIdx.y;
  int z = blockIdx.z;
  if (h >= L.hh || R * yp >= L.n[1]) return;
  V2 E = var2(fp, L.oe, L.half), G = var2(fp, L.og, L.half);
  const float* PB = fp + L.opb;
  unsigned own[R];
  float pb[R], xv[R], s0[R], s1[R], g0[R], g1[R];
  for (int k = 0; k < R; k++) {
    int y = R * yp + k;
    int x = 2 * h + ((c + y + z + (DIM == 3 ? 1 : 0)) & 1);
    Loc<DIM> l(L, x, y, z);
    own[k] = l.own;
    pb[k] = PB[l.own];
    s0[k] = s1[k] = xv[k] = 0.f;
    if (first != 1) {
      s0[k] = nsum<DIM>(E.v0, l);
      s1[k] = nsum<DIM>(E.v1, l);
      if (first == 0) xv[k] = E.v0[l.own];
    }
    g0[k] = G.v0[l.own];
    g1[k] = G.v1[l.own];
  }
  for (int k = 0; k < R; k++) {
    float r0, r1;
    newton_cell(L, pb[k], xv[k], s0[k], s1[k], g0[k], g1[k], r0, r1);
    E.v0[own[k]] = r0;
    E.v1[own[k]] = r1;
  }
}

// ---------------------------------------------------------------------------
// The same colour sweep (3D) with its rows staged in shared memory by bulk
// asynchronous copies (cp.async.bulk, completion counted on an mbarrier).
// A tile is kTileRows consecutive rows y of one plane z of the own colour; it
// needs the own rows of pb, g0, g1 (and e0 unless first) and the other
// colour's e0, e1 rows y-1..y+kTileRows at z and y..y+kTileRows-1 at z-1 and
// z+1 (periodic wrap).  Persistent CTAs walk the tiles plane by plane, the
// next tile's rows in flight while the current one is computed, so the
// memory system always has whole rows outstanding instead of one word per
// thread.  The cell update is k_bx_relax's (newton_cell); the six neighbours
// are summed left to right, where that adds the two z-neighbours as a
// pair, so the values agree to rounding, not bit for bit.
constexpr int kTileThreads = 256;
constexpr long long kWaitLimit = 1ll << 24;  // mbarrier polls before giving up

__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ bool mbar_wait(unsigned bar, unsigned parity) {
  for (long long it = 0; it < kWaitLimit; it++) {
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}

// floats of one stage: own pb, g0, g1, e0 (4 T rows), other e0/e1 at z
// (2 (T+2) rows), at z-1 and z+1 (4 T rows)
__host__ __device__ __forceinline__ int tile_stage_floats(int T, int hh) { return (10 * T + 4) * hh; }

// T rows per tile, NS stages (NS - 1 tiles in flight ahead of the one computed)
template <int T, int NS>
__global__ void __launch_bounds__(kTileThreads) k_bx_relax_tiled(float* __restrict__ fp, BoxLev L, int c, int first) {
  after_previous();
  extern __shared__ __align__(128) float tsm[];
  __shared__ __align__(8) unsigned long long bar[NS];
  const int hh = L.hh, n1 = L.n[1], n2 = L.n[2];
  const int SF = tile_stage_floats(T, hh);
  const int tiles_per_plane = n1 / T, ntiles = tiles_per_plane * n2;
  const unsigned rowb = (unsigned)hh * 4u;
  const long long half = L.half;
  // bases of the colour-split arrays (variable v, colour k): off + (2v+k)*half
  const float* E = fp + L.oe;
  const float* G = fp + L.og;
  const float* PB = fp + L.opb;
  const int o = 1 - c;  // the other colour
  if (threadIdx.x == 0) {
    for (int b = 0; b < NS; b++)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&bar[b])));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  // rows of a tile into stage buffer sb: consecutive rows of one array are
  // contiguous in memory, so each array's rows go as one bulk copy (two or
  // three where the rows wrap around the plane); thread 0 issues them
  auto issue = [&](int tile, int sb) {
    if (threadIdx.x != 0) return;
    int z = tile / tiles_per_plane, y0 = (tile % tiles_per_plane) * T;
    int nrows = first == 1 ? 3 * T : (first == 2 ? 3 * T + 2 * (T + 2) + 4 * T : 4 * T + 2 * (T + 2) + 4 * T);
    unsigned b = smem_addr(&bar[sb]);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(b), "r"((unsigned)nrows * rowb)
                 : "memory");
    float* base = tsm + sb * SF;
    // rows y .. y+n-1 (wrapping in the plane) of plane zz of array a -> slots from `slot`
    auto rows = [&](const float* a, int zz, int y, int n, int slot) {
      while (n > 0) {
        int yy = y < 0 ? y + n1 : (y >= n1 ? y - n1 : y);
        int run = n1 - yy < n ? n1 - yy : n;
        asm volatile(
            "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                smem_addr(base + (long long)slot * hh)),
            "l"(a + ((long long)zz * n1 + yy) * hh), "r"((unsigned)run * rowb), "r"(b)
            : "memory");
        y += run;
        n -= run;
        slot += run;
      }
    };
    rows(PB + (long long)c * half, z, y0, T, 0);
    rows(G + (long long)c * half, z, y0, T, T);
    rows(G + (long long)(2 + c) * half, z, y0, T, 2 * T);
    if (first == 0) rows(E + (long long)c * half, z, y0, T, 3 * T);
    if (first != 1) {
      int zm = z ? z - 1 : n2 - 1, zp = z + 1 < n2 ? z + 1 : 0;
      for (int v = 0; v < 2; v++) {
        const float* a = E + (long long)(2 * v + o) * half;
        rows(a, z, y0 - 1, T + 2, 4 * T + v * (T + 2));
        rows(a, zm, y0, T, 4 * T + 2 * (T + 2) + v * T);
        rows(a, zp, y0, T, 4 * T + 2 * (T + 2) + 2 * T + v * T);
      }
    }
  };
  int it = 0;
  int tile = blockIdx.x;
  for (int k = 0; k < NS - 1; k++)
    if (tile + k * (int)gridDim.x < ntiles) issue(tile + k * gridDim.x, k);
  bool ok = true;
  for (; tile < ntiles; tile += gridDim.x, it++) {
    int sb = it % NS;
    int next = tile + (NS - 1) * gridDim.x;  // its buffer was released by the barrier ending the last iteration
    if (next < ntiles) issue(next, (it + NS - 1) % NS);
    ok = mbar_wait(smem_addr(&bar[sb]), (unsigned)((it / NS) & 1)) && ok;
    const float* st = tsm + sb * SF;
    const float* sPB = st;
    const float* sG0 = st + T * hh;
    const float* sG1 = st + 2 * T * hh;
    const float* sE0 = st + 3 * T * hh;
    const float* sO0 = st + 4 * T * hh;          // other e0 at z, rows y0-1..y0+T
    const float* sO1 = sO0 + (T + 2) * hh;       // other e1 at z
    const float* sZ = sO1 + (T + 2) * hh;        // z-1: e0, e1; z+1: e0, e1 (T rows each)
    int z = tile / tiles_per_plane, y0 = (tile % tiles_per_plane) * T;
    for (int q = threadIdx.x; q < T * hh; q += kTileThreads) {
      int yl = q / hh, h = q - yl * hh;
      int y = y0 + yl;
      int bb = (c + y + z + 1) & 1;  // x = 2h + bb
      int xm = bb ? h : (h ? h - 1 : hh - 1);
      int xp = bb ? (h + 1 < hh ? h + 1 : 0) : h;
      float pb = sPB[q];
      float s0 = 0.f, s1 = 0.f, xv = 0.f;
      if (first != 1) {
        const float* a0 = sO0 + (yl + 1) * hh;
        const float* a1 = sO1 + (yl + 1) * hh;
        s0 = a0[xm] + a0[xp] + a0[h - hh] + a0[h + hh] + sZ[q] + sZ[2 * T * hh + q];
        s1 = a1[xm] + a1[xp] + a1[h - hh] + a1[h + hh] + sZ[T * hh + q] + sZ[3 * T * hh + q];
        if (first == 0) xv = sE0[q];
      }
      float r0, r1;
      newton_cell(L, pb, xv, s0, s1, sG0[q], sG1[q], r0, r1);
      if (!ok) r0 = r1 = __int_as_float(0x7fc00000);  // a copy that never landed: poison the sweep
      long long row = ((long long)z * n1 + y) * hh + h;
      float* Ew = fp + L.oe;
      Ew[(long long)c * half + row] = r0;
      Ew[(long long)(2 + c) * half + row] = r1;
    }
    __syncthreads();  // every thread is done with buffer sb before it is refilled
  }
  if (!ok)  // a wait gave up: give the copies still in flight a bounded time to land before the block exits
    for (int b = 0; b < NS; b++) mbar_wait(smem_addr(&bar[b]), 0u), mbar_wait(smem_addr(&bar[b]), 1u);
}

// ---------------------------------------------------------------------------
// One smoothing of a 3D level's V-cycle visit (nsmooth = 2: colour
// half-sweeps 0, 1, 0, 1) in one pass over memory.  A CTA owns a run of the
// planes of the y-tiles laid end to end (see SmoothSplit): for every tile of
// its run, the TY rows y0 .. y0+TY-1 of the planes z0 .. z1-1, for which it
// streams the planes z0-NS .. z1+NS-1
// through a ring of NS+3 shared-memory slots, each holding the four
// colour-split e arrays of rows y0-NS .. y0+TY+NS-1 of one plane (TMA tensor
// copies of four rows of one array, at row chunks wrapped around the plane).
// Once plane i has landed, stage
// s (half-sweep s) updates plane i-s: it needs the other colour of planes
// i-s-1 .. i-s+1 at stage s-1, which stage s-1 produced in this pass or the
// last.  Each stage's rows shrink by one at both ends (its neighbours must
// be at the previous stage), so stage NS leaves rows y0 .. y0+TY-1 final,
// and the planes outside z0 .. z1-1 are computed only as halo.  Colour
// updates read only the other colour and their own cell, so the result is
// the NS separate half-sweeps' bit for bit.  g and pb come from global
// memory into registers one plane ahead of the stage that uses them.  The
// output goes to a second e array (oe_out): the input rows of a tile's halo
// belong to other CTAs' outputs.  DRAM bytes per cell for NS = 4: 8 (e,
// none when fresh) + 8 (g) + 4 (pb) read, 8 written, against 4 x 18 for four
// separate half-sweeps.
constexpr int kSmStages = 4;      // half-sweeps per pass
constexpr int kSmThreads = 512;
constexpr int kSmMinPlanes = 16;  // fewest planes a CTA is made for (the halo costs 2 NS more)
constexpr int kSmMaxCtas = 256;
// CTA b smooths the planes start[b] .. start[b+1]-1 of the line in which plane
// z of y-tile t is t * n2 + z
struct SmoothSplit {
  int start[kSmMaxCtas + 1];
};

__host__ __device__ constexpr int smooth_slots(int ns) { return ns + 3; }  // planes i-ns-1 .. i, i+1 in flight
__host__ __device__ constexpr long long smooth_slot_floats(int ty, int hh, int ns = kSmStages) {
  return 4LL * (ty + 2 * ns) * hh;
}
__host__ __device__ constexpr int ilog2(int n) { return n <= 1 ? 0 : 1 + ilog2(n / 2); }

// CPT consecutive cells of a colour row as one vector access (4: float4,
// 2: float2)
template <int CPT>
__device__ __forceinline__ void ldv(const float* p, float* v) {
  if constexpr (CPT == 4) {
    const float4 t = *reinterpret_cast<const float4*>(p);
    v[0] = t.x, v[1] = t.y, v[2] = t.z, v[3] = t.w;
  } else {
    const float2 t = *reinterpret_cast<const float2*>(p);
    v[0] = t.x, v[1] = t.y;
  }
}
template <int CPT>
__device__ __forceinline__ void stv(float* p, const float* v) {
  if constexpr (CPT == 4) *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
  else *reinterpret_cast<float2*>(p) = make_float2(v[0], v[1]);
}

// TY rows a tile, HH cells a colour row, FRESH: the old e counts as zero (the
// finest level's pre-smoothing), NS stages, CPT consecutive cells of a row a
// thread, NT threads a CTA.  The library runs CPT = 4 at 512 threads (two
// cells a thread at 1024 threads measured no faster: the kernel is bound by
// its instructions, not by the warps it has to hide latency).
template <int TY, int HH, bool FRESH, int NS = kSmStages, int CPT = 4, int NT = kSmThreads>
__global__ void __launch_bounds__(NT, 1) k_bx_smooth(float* __restrict__ fp, BoxLev L, long long oe_out,
                                                   const __grid_constant__ SmoothSplit split,
                                                   const __grid_constant__ CUtensorMap emap) {
  after_previous();
  extern __shared__ __align__(128) float ssm[];
  constexpr int NSL = smooth_slots(NS);
  constexpr int R = TY + 2 * NS, AR = R * HH, SL = 4 * AR, LG = ilog2(HH);
  constexpr int W = HH / CPT;               // threads of a colour row: CPT consecutive cells each
  constexpr int RK = NT / W;                // rows between a thread's row segments
  constexpr int KQ = (R + RK - 1) / RK;     // row segments of a thread (the same rows in every stage)
  constexpr bool CARRY = CPT == 4;          // registers for the carried in-plane values
  static_assert((1 << LG) == HH && HH % 4 == 0 && RK % 2 == 0 && (CPT == 2 || CPT == 4), "rows of 2^k cells");
  static_assert(R % 4 == 0 && TY % 4 == 0, "slots fill in chunks of four rows");
  __shared__ __align__(8) unsigned long long bar[NSL];
  const int n1 = L.n[1], n2 = L.n[2];
  const unsigned half = (unsigned)L.half;  // a level's cells are fewer than 2^31
  int y0 = 0, z0 = 0, P = 0;  // the segment of one tile: local plane j is z0 - NS + j
  const float* G = fp + L.og;
  const float* PB = fp + L.opb;
  float* EO = fp + oe_out;
  auto wrap = [](int v, int n) { return v < 0 ? v + n : (v >= n ? v - n : v); };
  // this thread's cells hc .. hc+CPT-1 of rows rb + k RK: the same in every
  // stage, so that a stage's z+1 values are the ones the thread computed in
  // the stage before it, and no other thread writes what a stage reads in
  // the same pass but the rows y+-1 and the row neighbours beyond the
  // thread's cells, which were written in the pass before
  const int li = threadIdx.x % W, rb = threadIdx.x / W, hc = CPT * li;
  const int hm = (hc - 1) & (HH - 1), hp = (hc + CPT) & (HH - 1);  // the row's periodic wrap
  unsigned goff[KQ];  // the cells' offset within a plane of a colour-split array
  if (threadIdx.x == 0) {
    for (int b = 0; b < NSL; b++) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&bar[b])));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  // lane 0 of warps 0-3: the rows y0-NS .. y0+TY+NS-1 of the four e arrays
  // of local plane j into slot k, by tensor copies of four rows of one array
  // (emap: the input e as [array][z][y][h], a box of 4 x HH cells); warp w
  // copies the row chunks w, w+4, ..., whose start rows, wrapped around the
  // plane, are whole chunks (n1 is a multiple of 4); warp 0 arms the barrier
  // with the plane's bytes.  Nothing when fresh: the first half-sweeps count
  // the old e as zero.
  auto issue = [&](int j, int k) {
    const int w = threadIdx.x >> 5;
    if (FRESH || (threadIdx.x & 31) || w >= 4 || j >= P) return;
    const unsigned b = smem_addr(&bar[k]);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    if (w == 0)
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(b), "r"((unsigned)SL * 4u)
                   : "memory");
    const int zw = wrap(z0 - NS + j, n2);
    for (int ck = w; ck < R / 4; ck += 4) {
      const int yc = wrap(y0 - NS + 4 * ck, n1);
      for (int a = 0; a < 4; a++)
        asm volatile(
            "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], "
            "[%6];" ::"r"(smem_addr(ssm + k * SL + a * AR + ck * 4 * HH)),
            "l"(reinterpret_cast<unsigned long long>(&emap)), "r"(0), "r"(yc), "r"(zw), "r"(a), "r"(b)
            : "memory");
    }
  };
  // pb, g0, g1 of this thread's cells of stage s for the pass over local
  // plane j, in registers before that pass
  float v[NS][KQ][3][CPT];
  auto load = [&](int s, int j) {
    if (j < s || j > P - 1 - s) return;  // uniform over the CTA
    const unsigned c = (s - 1) & 1;
    const unsigned zoff = (unsigned)(wrap(z0 - NS + j, n2) * n1 * HH);
#pragma unroll
    for (int k = 0; k < KQ; k++) {
      const int r = rb + k * RK;
      if (r >= s && r <= R - 1 - s) {
        const unsigned gi = zoff + goff[k];
        ldv<CPT>(PB + (c * half + gi), v[s - 1][k][0]);
        ldv<CPT>(G + (c * half + gi), v[s - 1][k][1]);
        ldv<CPT>(G + ((2 + c) * half + gi), v[s - 1][k][2]);
      }
    }
  };
  // per stage, the other colour of the thread's cells in the plane after the
  // one last passed
  float cz[NS][CARRY ? KQ : 1][2][CPT];
  bool ok = true;
  int si = 0;               // the slot of plane i: the planes passed before it, of all segments, mod NSL
  unsigned phase = 0;       // its barrier's phase parity: those planes / NSL, & 1
  auto slot = [&](int d) {  // the slot of plane i - d (0 <= d < NSL)
    const int t = si - d;
    return t < 0 ? t + NSL : t;
  };
  const int end = split.start[blockIdx.x + 1];
  for (int p = split.start[blockIdx.x]; p < end; p += P - 2 * NS) {
    const int tile = p / n2;
    y0 = tile * TY, z0 = p - tile * n2;
    P = min(n2 - z0, end - p) + 2 * NS;
#pragma unroll
    for (int k = 0; k < KQ; k++) goff[k] = (unsigned)(wrap(y0 - NS + rb + k * RK, n1) * HH + hc);
    // the last barrier of the segment before lies behind the last reads of
    // these two slots (planes i-NS-2 and i-NS-1 of its last pass)
    issue(0, si);
    issue(1, si + 1 == NSL ? 0 : si + 1);
    for (int i = 0; i < P; i++) {
      if (!FRESH) ok = mbar_wait(smem_addr(&bar[si]), phase) && ok;
      float fw[KQ][2][CPT];  // the last stage's new values: the z+1 values of the next stage
#pragma unroll
      for (int s = 1; s <= NS; s++) {
        const int j = i - s;
        if (j >= s && j <= P - 1 - s) {  // uniform over the CTA
          const int c = (s - 1) & 1, o = 1 - c;
          const int first = FRESH ? (s <= 2 ? s : 0) : 0;
          // x = 2h + bb: the parity is the same for all of the thread's rows (RK is even)
          const int bb = (c + y0 - NS + rb + z0 - NS + j + 1) & 1;
          float* S = ssm + slot(s) * SL + (rb << LG);
          const float* Sm = ssm + slot(s + 1) * SL + (rb << LG);
          const float* Sp = ssm + slot(s - 1) * SL + (rb << LG);
#pragma unroll
          for (int k = 0; k < KQ; k++) {
            const int r = rb + k * RK;
            if (r >= s && r <= R - 1 - s) {
              const int ro = k * RK * HH;
              float s0[CPT], s1[CPT], xv[CPT];
#pragma unroll
              for (int q = 0; q < CPT; q++) s0[q] = s1[q] = xv[q] = 0.f;
              if (first != 1) {
#pragma unroll
                for (int var = 0; var < 2; var++) {
                  const int ao = (2 * var + o) * AR + ro;
                  float a[CPT], zp[CPT], zm[CPT], ym[CPT], yp[CPT];
                  // the other colour of this plane was the z+1 value of the
                  // pass over plane j-1, unchanged since
                  if (CARRY && j > s) {
#pragma unroll
                    for (int q = 0; q < CPT; q++) a[q] = cz[s - 1][CARRY ? k : 0][var][q];
                  } else {
                    ldv<CPT>(S + ao + hc, a);
                  }
                  if (s == 1) {
                    ldv<CPT>(Sp + ao + hc, zp);
                  } else {
#pragma unroll
                    for (int q = 0; q < CPT; q++) zp[q] = fw[k][var][q];
                  }
                  if (CARRY) {
#pragma unroll
                    for (int q = 0; q < CPT; q++) cz[s - 1][CARRY ? k : 0][var][q] = zp[q];
                  }
                  ldv<CPT>(Sm + ao + hc, zm);
                  ldv<CPT>(S + ao - HH + hc, ym);
                  ldv<CPT>(S + ao + HH + hc, yp);
                  // a[xm] + a[xp] with xm, xp = h, h+1 (bb = 1) or h-1, h (bb = 0)
                  const float edge = S[ao + (bb ? hp : hm)];
                  float* acc = var ? s1 : s0;
#pragma unroll
                  for (int q = 0; q < CPT; q++) {
                    const float lft = bb ? a[q] : (q ? a[q - 1] : edge);
                    const float rgt = bb ? (q + 1 < CPT ? a[q + 1] : edge) : a[q];
                    float t = lft + rgt + ym[q] + yp[q];
                    t += zm[q] + zp[q];
                    acc[q] = t;
                  }
                }
                if (first == 0) ldv<CPT>(S + c * AR + ro + hc, xv);
              }
              float r0[CPT], r1[CPT];
#pragma unroll
              for (int q = 0; q < CPT; q++) {
                newton_cell(L, v[s - 1][k][0][q], xv[q], s0[q], s1[q], v[s - 1][k][1][q], v[s - 1][k][2][q], r0[q],
                            r1[q]);
                if (!ok) r0[q] = r1[q] = nanf("");  // a copy that never landed: poison the pass
                fw[k][0][q] = r0[q], fw[k][1][q] = r1[q];
              }
              stv<CPT>(S + c * AR + ro + hc, r0);
              stv<CPT>(S + (2 + c) * AR + ro + hc, r1);
            }
          }
        }
        load(s, i + 1 - s);  // the next pass's cells of this stage, in flight while the others compute
      }
      __syncthreads();  // rows y+-1 of this pass are read by the next; the slot below is free
      issue(i + 2, slot(NSL - 2));  // plane i + 2 into the slot of plane i - NS - 1, which stage NS read last
      const int j = i - NS;
      if (j >= NS && j <= P - 1 - NS) {  // plane j is final: rows NS .. NS+TY-1 of the slot
        const float* S = ssm + slot(NS) * SL + NS * HH;
        float* D = EO + (unsigned)(((z0 - NS + j) * n1 + y0) * HH);
        constexpr int n4 = (TY * HH) >> 2;
#pragma unroll
        for (int q = threadIdx.x; q < 4 * n4; q += NT) {
          const int a = q / n4, t = q - a * n4;
          reinterpret_cast<float4*>(D + (unsigned)a * half)[t] = reinterpret_cast<const float4*>(S + a * AR)[t];
        }
      }
      if (++si == NSL) si = 0, phase ^= 1u;
    }
  }
  if (!ok)  // a wait gave up: give the copies still in flight a bounded time to land before the block exits
    for (int b = 0; b < NSL; b++) mbar_wait(smem_addr(&bar[b]), 0u), mbar_wait(smem_addr(&bar[b]), 1u);
}

// RestrictSolution and the fine half of CoarseLoadingFunction in one pass
// over the fine cells: coarse e = ec = R(e), coarse pb = R(pb) and coarse
// g = R(g - M(e)); the coarse operator M_c(ec) needs the neighbours' ec, so
// k_bx_coarse_op adds it in a second (coarse-sized) pass.  2D:
__global__ void __launch_bounds__(256, 6) k_bx_restrict_load(float* __restrict__ fp, BoxLev F, BoxLev C) {
  after_previous();
  const int X = blockIdx.x * blockDim.x + threadIdx.x, Y = blockIdx.y * blockDim.y + threadIdx.y;
  if (X >= C.n[0] || Y >= C.n[1]) return;
  V2 Ef = var2(fp, F.oe, F.half), Gf = var2(fp, F.og, F.half);
  const float* PBf = fp + F.opb;
  float s0 = 0.f, s1 = 0.f, s2 = 0.f, R0 = 0.f, R1 = 0.f;
  for (int dy = 0; dy < 2; dy++)
    for (int dx = 0; dx < 2; dx++) {
      Loc<2> l(F, 2 * X + dx, 2 * Y + dy, 0);
      float pb = PBf[l.own];
      s0 += Ef.v0[l.own];
      s1 += Ef.v1[l.own];
      s2 += pb;
      float m0, m1;
      mop<2>(Ef, F, l, pb, m0, m1);
      R0 += Gf.v0[l.own] - m0;
      R1 += Gf.v1[l.own] - m1;
    }
  const float w = 0.25f;
  Loc<2> lc(C, X, Y, 0);
  V2 Ec = var2(fp, C.oe, C.half), ECc = var2(fp, C.oec, C.half), Gc = var2(fp, C.og, C.half);
  Ec.v0[lc.own] = ECc.v0[lc.own] = s0 * w;
  Ec.v1[lc.own] = ECc.v1[lc.own] = s1 * w;
  fp[C.opb + lc.own] = s2 * w;
  Gc.v0[lc.own] = R0 * w;
  Gc.v1[lc.own] = R1 * w;
}

// 3D: a thread owns two coarse cells of a row, whose fine cells are, in each
// colour's array, two consecutive values of four rows: it loads every value
// once, as a vector (72 vectors and 16 single ones for what cell by cell are
// 272 loads).  The pass waits for memory (cell by cell at 40 registers it took
// 135 us at 256^3 against 50 us for its bytes), so that fewer and wider loads,
// more of them in flight, are what counts: 200.6 -> 218.7 steps/s of 256^3
// (bench.py --steps 20 --warmup 5) with five CTAs of 128 threads an SM at 96
// registers; over a shorter run 234, at 64 registers 225, with four cells a
// thread at 128 registers 232.  The sums keep the order of the cells, and the
// bits.
constexpr int kRestrictThreads = 128;
constexpr int kRestrictCells = 2;  // coarse cells a thread; a level's extents are even
__global__ void __launch_bounds__(kRestrictThreads, 5) k_bx_restrict_rows(float* __restrict__ fp, BoxLev F, BoxLev C) {
  after_previous();
  constexpr int CPT = kRestrictCells;
  const int X = CPT * (int)(blockIdx.x * blockDim.x + threadIdx.x), Y = blockIdx.y * blockDim.y + threadIdx.y;
  const int Z = blockIdx.z;
  if (X >= C.n[0] || Y >= C.n[1]) return;
  const unsigned hh = (unsigned)F.hh, n1 = (unsigned)F.n[1], n2 = (unsigned)F.n[2], half = (unsigned)F.half;
  const unsigned h = (unsigned)X;  // fine x = 2 X + dx is position X of its colour's row
  const unsigned hl = h ? h - 1 : hh - 1, hr = h + CPT < hh ? h + CPT : 0u;
  const unsigned y0 = 2u * (unsigned)Y, z0 = 2u * (unsigned)Z;
  // the rows below and above the cell's two in y and z
  const unsigned yo[2] = {y0 ? y0 - 1 : n1 - 1, y0 + 2 < n1 ? y0 + 2 : 0u};
  const unsigned zo[2] = {z0 ? z0 - 1 : n2 - 1, z0 + 2 < n2 ? z0 + 2 : 0u};
  const float* const E = fp + F.oe;
  const float* const G = fp + F.og;
  const float* const PB = fp + F.opb;
  float e[2][2][2][2][CPT];  // [variable][colour][dz][dy]
#pragma unroll
  for (int dz = 0; dz < 2; dz++)
#pragma unroll
    for (int dy = 0; dy < 2; dy++)
#pragma unroll
      for (int a = 0; a < 4; a++)
        ldv<CPT>(E + (a * half + ((z0 + dz) * n1 + y0 + dy) * hh + h), e[a >> 1][a & 1][dz][dy]);
  float t0[CPT], t1[CPT], t2[CPT], R0[CPT], R1[CPT];
#pragma unroll
  for (int q = 0; q < CPT; q++) t0[q] = t1[q] = t2[q] = R0[q] = R1[q] = 0.f;
#pragma unroll
  for (int dz = 0; dz < 2; dz++)
#pragma unroll
    for (int dy = 0; dy < 2; dy++) {
      const unsigned r = ((z0 + dz) * n1 + y0 + dy) * hh;
      const unsigned ry = ((z0 + dz) * n1 + yo[dy]) * hh + h, rz = (zo[dz] * n1 + y0 + dy) * hh + h;
      const int c0 = (dy + dz + 1) & 1;  // the colour of the cells dx = 0 (2X, 2Y and 2Z are even)
      float oy[2][2][CPT], oz[2][2][CPT], pb[2][CPT], g[2][2][CPT], edge[2][2];
#pragma unroll
      for (int a = 0; a < 4; a++) {
        ldv<CPT>(E + (a * half + ry), oy[a >> 1][a & 1]);
        ldv<CPT>(E + (a * half + rz), oz[a >> 1][a & 1]);
        ldv<CPT>(G + (a * half + r + h), g[a >> 1][a & 1]);
      }
#pragma unroll
      for (int v = 0; v < 2; v++) {
        ldv<CPT>(PB + (v * half + r + h), pb[v]);
        edge[v][0] = E[(2 * v + 1 - c0) * half + r + hl];
        edge[v][1] = E[(2 * v + c0) * half + r + hr];
      }
#pragma unroll
      for (int dx = 0; dx < 2; dx++) {
        const int c = (c0 + dx) & 1, o = 1 - c;
#pragma unroll
        for (int q = 0; q < CPT; q++) {
          float s[2];
#pragma unroll
          for (int v = 0; v < 2; v++) {
            const float* w = e[v][o][dz][dy];
            const float xm = dx ? w[q] : (q ? w[q ? q - 1 : 0] : edge[v][0]);
            const float xp = dx ? (q + 1 < CPT ? w[q + 1 < CPT ? q + 1 : 0] : edge[v][1]) : w[q];
            const float ym = dy ? e[v][o][dz][0][q] : oy[v][o][q], yp = dy ? oy[v][o][q] : e[v][o][dz][1][q];
            const float zm = dz ? e[v][o][0][dy][q] : oz[v][o][q], zp = dz ? oz[v][o][q] : e[v][o][1][dy][q];
            s[v] = xm + xp + ym + yp;
            s[v] += zm + zp;
          }
          const float x = e[0][c][dz][dy][q], y = e[1][c][dz][dy][q];
          float m0, m1;
          mop_cell<3>(F, x, y, pb[c][q], s[0], s[1], m0, m1);
          t0[q] += x;
          t1[q] += y;
          t2[q] += pb[c][q];
          R0[q] += g[0][c][q] - m0;
          R1[q] += g[1][c][q] - m1;
        }
      }
    }
  const float w = 0.125f;
  const unsigned ch = (unsigned)C.half, cr = ((unsigned)Z * (unsigned)C.n[1] + (unsigned)Y) * (unsigned)C.hh;
#pragma unroll
  for (int q = 0; q < CPT; q++) {
    const unsigned i = (colour<3>(X + q, Y, Z) ? ch : 0u) + cr + ((unsigned)(X + q) >> 1);
    fp[C.oe + i] = fp[C.oec + i] = t0[q] * w;
    fp[C.oe + 2 * ch + i] = fp[C.oec + 2 * ch + i] = t1[q] * w;
    fp[C.opb + i] = t2[q] * w;
    fp[C.og + i] = R0[q] * w;
    fp[C.og + 2 * ch + i] = R1[q] * w;
  }
}
// coarse g += M_c(ec), the coarse operator on the restricted correction
template <int DIM>
__global__ void __launch_bounds__(256) k_bx_coarse_op(float* __restrict__ fp, BoxLev C) {
  after_previous();
  int X = blockIdx.x * blockDim.x + threadIdx.x;
  int Y = blockIdx.y * blockDim.y + threadIdx.y;
  if (X >= C.n[0] || Y >= C.n[1]) return;
  Loc<DIM> lc(C, X, Y, blockIdx.z);
  V2 ECc = var2(fp, C.oec, C.half), Gc = var2(fp, C.og, C.half);
  float g0 = Gc.v0[lc.own], g1 = Gc.v1[lc.own];
  float m0, m1;
  mop<DIM>(ECc, C, lc, fp[C.opb + lc.own], m0, m1);
  Gc.v0[lc.own] = g0 + m0;
  Gc.v1[lc.own] = g1 + m1;
}

// CorrectFine on e: e_fine += P(e_c - ec), per-direction (3,1)/4 weights
// (Bi/TriLinProlongationP1, gridutilities.f90:156-195, :510-566).  Thread T
// (per dimension 0..nc-1) owns fine cells 2T-1 (wrapped) and 2T, between
// coarse cells T-1 (wrapped) and T.
template <int DIM>
__device__ __forceinline__ void prolong_at(float* __restrict__ fp, const BoxLev& F, const BoxLev& C, int T0, int T1,
                                           int T2) {
  const int T[3] = {T0, T1, T2};
  int cx[2][3], fx[2][3];
  for (int d = 0; d < 3; d++) {
    int n = C.n[d];
    cx[0][d] = T[d] ? T[d] - 1 : n - 1;
    cx[1][d] = T[d];
    fx[0][d] = T[d] ? 2 * T[d] - 1 : 2 * n - 1;
    fx[1][d] = 2 * T[d];
  }
  constexpr int NZ = DIM == 3 ? 2 : 1;
  V2 Ec = var2(fp, C.oe, C.half), ECc = var2(fp, C.oec, C.half), Ef = var2(fp, F.oe, F.half);
  // corrections e_c - ec at the 2x2(x2) coarse corners, both variables
  float a[2][NZ][2][2];
  for (int dz = 0; dz < NZ; dz++)
    for (int dy = 0; dy < 2; dy++)
      for (int dx = 0; dx < 2; dx++) {
        Loc<DIM> l(C, cx[dx][0], cx[dy][1], DIM == 3 ? cx[dz][2] : 0);
        a[0][dz][dy][dx] = Ec.v0[l.own] - ECc.v0[l.own];
        a[1][dz][dy][dx] = Ec.v1[l.own] - ECc.v1[l.own];
      }
  // weight 3/4 on the near coarse cell (f = 0: the first, f = 1: the second)
  auto w1 = [](float lo, float hi, int f) { return f == 0 ? 3.0f * lo + hi : lo + 3.0f * hi; };
  // every fine value is loaded before the first store, so the loads of one
  // thread are in flight together (a store to fp could alias a later load)
  constexpr int NF = 4 * NZ;
  unsigned own[NF];
  float val[NF][2];
  for (int m = 0; m < NF; m++) {
    int fxi = m & 1, fy = (m >> 1) & 1, fz = m >> 2;
    Loc<DIM> l(F, fx[fxi][0], fx[fy][1], DIM == 3 ? fx[fz][2] : 0);
    own[m] = l.own;
    val[m][0] = Ef.v0[l.own];
    val[m][1] = Ef.v1[l.own];
  }
  for (int m = 0; m < NF; m++) {
    int fxi = m & 1, fy = (m >> 1) & 1, fz = m >> 2;
    for (int v = 0; v < 2; v++) {
      float r0 = w1(w1(a[v][0][0][0], a[v][0][0][1], fxi), w1(a[v][0][1][0], a[v][0][1][1], fxi), fy);
      float add;
      if (DIM == 2) {
        add = r0 * (1.0f / 16.0f);
      } else {
        float r1 =
            w1(w1(a[v][NZ - 1][0][0], a[v][NZ - 1][0][1], fxi), w1(a[v][NZ - 1][1][0], a[v][NZ - 1][1][1], fxi), fy);
        add = w1(r0, r1, fz) * (1.0f / 64.0f);
      }
      val[m][v] += add;
    }
  }
  for (int m = 0; m < NF; m++) {
    Ef.v0[own[m]] = val[m][0];
    Ef.v1[own[m]] = val[m][1];
  }
}
template <int DIM>
__global__ void __launch_bounds__(256) k_bx_prolong(float* __restrict__ fp, BoxLev F, BoxLev C) {
  after_previous();
  int X = blockIdx.x * blockDim.x + threadIdx.x;
  int Y = blockIdx.y * blockDim.y + threadIdx.y;
  if (X < C.n[0] && Y < C.n[1]) prolong_at<DIM>(fp, F, C, X, Y, blockIdx.z);
}

// ---------------------------------------------------------------------------
// The coarse levels of the V-cycle in one launch of a thread-block cluster.
// Every CTA holds a slab of rows (the slowest dimension) of each level in
// shared memory, in natural order with one halo row at each side of e and ec;
// a CTA writes its boundary rows into its neighbours' halos as it computes
// them (distributed shared memory), so all reads are local and a sweep costs
// one cluster barrier.  Levels too small to share out are CTA 0's, or every
// second, fourth, .. CTA's (fold) where a CTA 0 would have more pairs than
// threads to hold them.
//
// A thread owns pairs of x-neighbours (2h, 2h+1), one cell of each colour,
// and keeps their e, g and pb in registers through a smoothing: a sweep reads
// the five (2D: three) neighbours outside the pair, updates and stores.  What
// surrounds the sweeps runs on the same registers: on the way down the
// coarse equation's M_c(ec) is added to g at the start and the residual
// g - M(e) that the coarse level averages is formed at the end; on the way up
// the prolonged correction is added at the start and e - ec, which the finer
// level prolongs, is left in ec at the end.
//
// Bound by latency: about 60 instructions a sweep and pair, a barrier of the
// cluster (0.3-0.5 us) or of the CTA (0.06 us), and on the coarsest level the
// FP64 unit, which takes 64 cycles a warp instruction however few lanes work.
// It took the place of one CTA on the levels up to 8192 cells (38 us for
// 64^2 .. 2^2) with a launch per sweep above: ten steps at 128^2 7.8 -> 5.95
// ms, five at 64^3 4.65 -> 4.15 ms, eight at 32^2 3.01 -> 2.68 ms, the same
// bits.
// 512 threads leave 128 registers, which do not hold two pairs' state in every
// form: spill stores and loads of 68 and 140 bytes a thread in 2D, 284 and 504
// in 3D (k_bx_solve, with its own state beside: 468 and 776, 900 and 1276),
// one instruction in fifty of k_bx_cycle, one in twenty of k_bx_solve.
struct CycLev {
  int n0, n1, N;       // extents (n1: 3D), rows
  int maxr;            // rows a CTA holds at most
  int mul, down;       // rows per row of the partition: mul / 2^down (mul 0: CTA 0 alone)
  int fold;            // every 2^fold-th CTA holds the level
  int e, ec, g, pb;    // starts in shared memory (floats)
  int by_colour;       // order of the restriction's sums (see cyc_smooth)
  float c0, c1, tmp3, a12;
  UniDiv hx, d1, hc, dc1;  // divisors: pairs of a row, n1, coarse cells of a row, coarse n1
};
struct Cyc {
  CycLev L[kNLev];     // finest first
  int row0[17];        // CTA r's first row of the level with mul = 1, down = 0 (the last: its rows)
  int nl, ctas, nsmooth, scratch;
  double cd[4];        // the coarsest level's coefficients in FP64
};
constexpr int kCycThreads = 512, kCycPairs = 2;  // threads of a CTA, most pairs a thread holds
extern __shared__ __align__(16) float csm[];

// This CTA's part of a level.
struct Slab {
  int n0, n1, N, r0, nr;
  int plane, var, ivar;  // floats of a row's plane, of a variable with halos, of an interior variable
  bool shared;
  int lo, hi, lo_rows;   // neighbours (around the domain) and the rows of the one below
  float *e, *ec, *g, *pb;
  float* base;           // the start of its CTA's shared memory
};
// A level's geometry as this CTA sees it, worked out once a launch and kept in
// shared memory: each smoothing starts from it.
struct __align__(16) SlabInfo {
  int n0, n1, N, r0;
  int nr, lo, hi, lo_rows;
  int e, ec, g, pb;
  int own, shared, maxr, workers;  // own: the CTA that holds this one's rows
};
constexpr int kCoarsePairs2 = 64;  // cyc_coarsest: most pairs that get two lanes each
template <int DIM>
__device__ __forceinline__ void slab_info(const Cyc& A, SlabInfo* info, int rank, int t, int nt) {
  if (t >= A.nl) return;
  const CycLev& L = A.L[t];
  SlabInfo S;
  S.n0 = L.n0, S.n1 = L.n1, S.N = L.N, S.r0 = 0, S.nr = L.N;
  S.lo = S.hi = 0, S.lo_rows = L.N;
  S.own = 0, S.shared = L.mul != 0, S.maxr = L.maxr;
  if (S.shared) {
    const int st = 1 << L.fold;  // CTAs st apart hold the level
    S.own = rank & -st;
    auto row = [&](int r) { return (A.row0[r] * L.mul) >> L.down; };
    S.r0 = row(S.own);
    S.nr = row(S.own + st) - S.r0;
    S.lo = S.own ? S.own - st : A.ctas - st;
    S.hi = S.own + st < A.ctas ? S.own + st : 0;
    S.lo_rows = row(S.lo + st) - row(S.lo);
  }
  S.e = L.e, S.ec = L.ec, S.g = L.g, S.pb = L.pb;
  // threads that work on it; coarser levels have no more than finer ones
  int units = (L.n0 >> 1) * (DIM == 3 ? L.n1 : 1) * L.maxr;
  if (t == A.nl - 1 && units <= kCoarsePairs2) units *= 2;
  S.workers = min(nt, (units + 31) & ~31);
  info[t] = S;
}
template <int DIM, bool REMOTE>
__device__ __forceinline__ Slab slab(const SlabInfo* info, int x, int rank) {
  const SlabInfo I = info[x];
  Slab S;
  S.n0 = I.n0, S.n1 = I.n1, S.N = I.N, S.r0 = I.r0, S.nr = I.nr;
  S.lo = I.lo, S.hi = I.hi, S.lo_rows = I.lo_rows;
  S.shared = I.shared != 0;
  S.plane = DIM == 3 ? I.n0 * I.n1 : I.n0;
  S.var = S.plane * (I.maxr + 2);
  S.ivar = S.plane * I.maxr;
  float* sm = csm;
  if (REMOTE && I.own != rank) sm = uni::on_rank(sm, I.own);
  S.base = sm;
  S.e = sm + I.e, S.ec = sm + I.ec, S.g = sm + I.g, S.pb = sm + I.pb;
  return S;
}

// Where a value of a halo array at local row `row` of a slab goes besides
// its own place: rows 1 and nr of a shared level into the neighbours' halos.
// (A level one CTA holds wraps its rows when read.)
struct HaloOut {
  float *lo, *hi;   // the array in the neighbours' shared memory
  int dlo, dhi;     // from a cell of row 1 (nr) to its image there
};
__device__ __forceinline__ HaloOut halo_out(const Slab& S, float* a) {
  HaloOut h{nullptr, nullptr, 0, 0};
  if (S.shared) {
    float* const mine = csm + (a - S.base);  // the array's place in every CTA
    h.lo = uni::on_rank(mine, S.lo);
    h.hi = uni::on_rank(mine, S.hi);
    h.dlo = S.lo_rows * S.plane;
    h.dhi = -S.nr * S.plane;
  }
  return h;
}
__device__ __forceinline__ void halo_put(const Slab& S, const HaloOut& h, int row, int at, float v) {
  if (!S.shared) return;
  if (row == 1) h.lo[at + h.dlo] = v;
  if (row == S.nr) h.hi[at + h.dhi] = v;
}

// A pair of cells (2h, 2h+1) of local row `row` (and y): its place in the
// halo arrays and the interior ones, the steps to the x-neighbours beyond the
// pair and to the other rows, and which of its cells has colour 0.
struct Pair {
  int at, in, row;
  int xl, xr, ym, yp, rm, rp;
  int b0;  // the colour-0 cell is at at + b0
};
template <int DIM>
__device__ __forceinline__ Pair pair_of(const Slab& S, const CycLev& L, int u) {
  Pair p;
  int r, h, y = 0, k;
  uni::fdivmod(u, L.hx, r, h);
  if (DIM == 3) uni::fdivmod(r, L.d1, k, y);
  else k = r;
  p.row = k + 1;
  const int base = DIM == 3 ? y * S.n0 + 2 * h : 2 * h;
  p.at = p.row * S.plane + base;
  p.in = k * S.plane + base;
  p.xl = h ? -1 : S.n0 - 1;
  p.xr = 2 * h + 2 < S.n0 ? 1 : 1 - S.n0;
  p.ym = y ? -S.n0 : (S.n1 - 1) * S.n0;
  p.yp = y + 1 < S.n1 ? S.n0 : -(S.n1 - 1) * S.n0;
  p.rm = S.shared || k ? -S.plane : (S.nr - 1) * S.plane;
  p.rp = S.shared || k + 1 < S.nr ? S.plane : -(S.nr - 1) * S.plane;
  p.b0 = (y + k + S.r0 + (DIM == 3 ? 1 : 0)) & 1;
  return p;
}
// sum over the neighbours of the pair's cell at at + b, `other` the pair's other cell
template <int DIM, typename T>
__device__ __forceinline__ T pair_sum(const float* a, const Pair& p, int b, T other) {
  const float* c = a + p.at + b;
  T s = T(b ? c[p.xr] : c[p.xl]) + other;
  if (DIM == 3) {
    s = s + T(c[p.ym]) + T(c[p.yp]);
    s += T(c[p.rm]) + T(c[p.rp]);
  } else {
    s = s + T(c[p.rm]) + T(c[p.rp]);
  }
  return s;
}

// What a smoothing does before its sweeps and after them.
enum CycBegin { kTop = 0, kDown = 1, kUp = 2 };

// One smoothing of this CTA's slab of level x (see above), K pairs a thread.
// sync: the level's barrier; local: that of this CTA's nt threads on it.  C: the
// parent level's slab.  The caller's
// barrier follows the call.
template <int DIM, int K, typename F, typename G>
__device__ __forceinline__ void cyc_smooth(const Cyc& A, int x, const Slab& S, const Slab& C, int begin, bool restrict_,
                                           bool emit, int t, int nt, F&& sync, G&& local) {
  const CycLev& L = A.L[x];
  const int units = (S.n0 >> 1) * (DIM == 3 ? S.n1 : 1) * S.nr;
  float *E0 = S.e, *E1 = S.e + S.var;
  const HaloOut H0 = halo_out(S, E0), H1 = halo_out(S, E1);
  // the pair's cells by colour, so that a sweep selects nothing: their places,
  // the step to the x-neighbour beyond the pair, e, g, pb ([..][variable])
  Pair p[K];
  bool on[K];
  int at[K][2], xo[K][2];
  float e[K][2][2], g[K][2][2], pb[K][2];
#pragma unroll
  for (int q = 0; q < K; q++) {
    on[q] = t + q * nt < units;
    if (!on[q]) continue;
    p[q] = pair_of<DIM>(S, L, t + q * nt);
#pragma unroll
    for (int c = 0; c < 2; c++) {
      const int b = p[q].b0 ^ c, in = p[q].in + b;
      at[q][c] = p[q].at + b;
      xo[q][c] = b ? p[q].xr : p[q].xl;
      e[q][c][0] = E0[at[q][c]];
      e[q][c][1] = E1[at[q][c]];
      g[q][c][0] = S.g[in];
      g[q][c][1] = S.g[S.ivar + in];
      pb[q][c] = S.pb[in];
    }
  }
  auto sum = [&](const float* a, int q, int c, float other) {  // pair_sum
    const float* w = a + at[q][c];
    float s = w[xo[q][c]] + other;
    if (DIM == 3) {
      s = s + w[p[q].ym] + w[p[q].yp];
      s += w[p[q].rm] + w[p[q].rp];
    } else {
      s = s + w[p[q].rm] + w[p[q].rp];
    }
    return s;
  };
  const float kc = DIM == 2 ? 4.0f : 6.0f;
  auto mop_cell = [&](int q, int c, float& m0, float& m1) {  // M(e) (mop)
    const float xx = e[q][c][0], y = e[q][c][1];
    const float s0 = sum(E0, q, c, e[q][1 - c][0]);
    const float s1 = sum(E1, q, c, e[q][1 - c][1]);
    m0 = xx - L.c0 * (s1 - kc * y);
    m1 = y - xx * (3.0f * pb[q][c] * (pb[q][c] + xx) + xx * xx) + L.c1 * (s0 - kc * xx);
  };
  if (begin == kDown) {  // g = R(g - M(e)) (left by the finer level) + M_c(ec); e is ec here
#pragma unroll
    for (int q = 0; q < K; q++)
      if (on[q]) {
        float m[2][2];
#pragma unroll
        for (int c = 0; c < 2; c++) mop_cell(q, c, m[c][0], m[c][1]);
#pragma unroll
        for (int c = 0; c < 2; c++)
#pragma unroll
          for (int v = 0; v < 2; v++) {
            g[q][c][v] += m[c][v];
            S.g[v * S.ivar + at[q][c] - S.plane] = g[q][c][v];
          }
      }
    sync();
  }
  if (begin == kUp) {  // e += P(e_c - ec), the difference in the parent's ec
#pragma unroll
    for (int q = 0; q < K; q++)
      if (on[q]) {
        const int u = t + q * nt;
        int r, h, y = 0, k;
        uni::fdivmod(u, L.hx, r, h);
        if (DIM == 3) uni::fdivmod(r, L.d1, k, y);
        else k = r;
        const int z = k + S.r0;  // global row
        // coarse columns h-1, h, h+1 and, per dimension, the near and the far coarse cell
        const int xm = h ? h - 1 : C.n0 - 1, xp = h + 1 < C.n0 ? h + 1 : 0;
        const int yn = y >> 1, yf = (y & 1) ? (yn + 1 < C.n1 ? yn + 1 : 0) : (yn ? yn - 1 : C.n1 - 1);
        // local coarse rows (row 1 is the slab's first; shared slabs have halo rows)
        const int zn = (z >> 1) - C.r0 + 1;
        int zf = (z & 1) ? zn + 1 : zn - 1;
        if (!C.shared) zf = zf < 1 ? C.nr : (zf > C.nr ? 1 : zf);
        auto xstage = [&](const float* a, int yy, int zz, float& lo, float& hi) {
          const float* c = a + zz * C.plane + (DIM == 3 ? yy * C.n0 : 0);
          const float v0 = c[xm], v1 = c[h], v2 = c[xp];
          lo = v0 + 3.0f * v1;  // cell 2h
          hi = 3.0f * v1 + v2;  // cell 2h+1
        };
#pragma unroll
        for (int v = 0; v < 2; v++) {
          const float* a = C.ec + v * C.var;
          float lo, hi, l2, h2;
          if (DIM == 3) {
            float a0, a1, b0, b1;
            xstage(a, yn, zn, a0, a1);
            xstage(a, yf, zn, b0, b1);
            lo = 3.0f * a0 + b0, hi = 3.0f * a1 + b1;
            xstage(a, yn, zf, a0, a1);
            xstage(a, yf, zf, b0, b1);
            l2 = 3.0f * a0 + b0, h2 = 3.0f * a1 + b1;
          } else {
            xstage(a, 0, zn, lo, hi);
            xstage(a, 0, zf, l2, h2);
          }
          const float w = DIM == 3 ? 1.0f / 64.0f : 1.0f / 16.0f;
          const float elo = p[q].b0 ? e[q][1][v] : e[q][0][v], ehi = p[q].b0 ? e[q][0][v] : e[q][1][v];
          const float nlo = elo + (3.0f * lo + l2) * w, nhi = ehi + (3.0f * hi + h2) * w;
          e[q][0][v] = p[q].b0 ? nhi : nlo;
          e[q][1][v] = p[q].b0 ? nlo : nhi;
#pragma unroll
          for (int c = 0; c < 2; c++) {
            (v ? E1 : E0)[at[q][c]] = e[q][c][v];
            halo_put(S, v ? H1 : H0, p[q].row, at[q][c], e[q][c][v]);
          }
        }
      }
    sync();
  }
  for (int s = 0; s < A.nsmooth; s++)
#pragma unroll
    for (int c = 0; c < 2; c++) {
#pragma unroll
      for (int q = 0; q < K; q++)
        if (on[q]) {
          const float s0 = sum(E0, q, c, e[q][1 - c][0]), s1 = sum(E1, q, c, e[q][1 - c][1]);
          newton_cell(L.c0, L.c1, L.tmp3, L.a12, pb[q][c], e[q][c][0], s0, s1, g[q][c][0], g[q][c][1], e[q][c][0],
                      e[q][c][1]);
          E0[at[q][c]] = e[q][c][0];
          E1[at[q][c]] = e[q][c][1];
          halo_put(S, H0, p[q].row, at[q][c], e[q][c][0]);
          halo_put(S, H1, p[q].row, at[q][c], e[q][c][1]);
        }
      if (c == 0 || s + 1 < A.nsmooth || restrict_) sync();
    }
  if (emit) {  // ec = e - ec, for the finer level's prolongation
    const HaloOut C0 = halo_out(S, S.ec), C1 = halo_out(S, S.ec + S.var);
#pragma unroll
    for (int q = 0; q < K; q++)
      if (on[q])
#pragma unroll
        for (int c = 0; c < 2; c++)
#pragma unroll
          for (int v = 0; v < 2; v++) {
            float* d = S.ec + v * S.var + at[q][c];
            const float w = e[q][c][v] - *d;
            *d = w;
            halo_put(S, v ? C1 : C0, p[q].row, at[q][c], w);
          }
  }
  if (!restrict_) return;
  // the residual g - M(e), which the coarse cells average
  float* const sc = csm + A.scratch;
#pragma unroll
  for (int q = 0; q < K; q++)
    if (on[q]) {
#pragma unroll
      for (int c = 0; c < 2; c++) {
        float m0, m1;
        mop_cell(q, c, m0, m1);
        sc[at[q][c] - S.plane] = g[q][c][0] - m0;
        sc[S.ivar + at[q][c] - S.plane] = g[q][c][1] - m1;
      }
    }
  local();
  // RestrictSolution and the fine half of CoarseLoadingFunction
  const int cu = units >> (DIM == 3 ? 2 : 1);
  const float w = DIM == 3 ? 0.125f : 0.25f;
  const HaloOut C0 = halo_out(C, C.e), C1 = halo_out(C, C.e + C.var);
  const HaloOut D0 = halo_out(C, C.ec), D1 = halo_out(C, C.ec + C.var);
  for (int u = t; u < cu; u += nt) {
    int r, X, Y = 0, Z;
    uni::fdivmod(u, L.hc, r, X);
    if (DIM == 3) uni::fdivmod(r, L.dc1, Z, Y);
    else Z = r;
    float a[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int dz = 0; dz < 2; dz++)
#pragma unroll
      for (int dy = 0; dy < (DIM == 3 ? 2 : 1); dy++) {
        const int k = 2 * Z + dz, y = 2 * Y + dy;
        const int in = k * S.plane + (DIM == 3 ? y * S.n0 : 0) + 2 * X, at = in + S.plane;
        // a row's two cells of e and pb: colour 0 first on small levels, else left to right
        const int b = L.by_colour ? (y + k + S.r0 + (DIM == 3 ? 1 : 0)) & 1 : 0;
        a[0] += E0[at + b];
        a[0] += E0[at + 1 - b];
        a[1] += E1[at + b];
        a[1] += E1[at + 1 - b];
        a[2] += S.pb[in + b];
        a[2] += S.pb[in + 1 - b];
        a[3] += sc[in];
        a[3] += sc[in + 1];
        a[4] += sc[S.ivar + in];
        a[4] += sc[S.ivar + in + 1];
      }
#pragma unroll
    for (int v = 0; v < 5; v++) a[v] *= w;
    const int row = Z + (S.r0 >> 1) - C.r0 + 1;
    const int in = (row - 1) * C.plane + (DIM == 3 ? Y * C.n0 : 0) + X, at = in + C.plane;
    C.e[at] = a[0];
    C.e[C.var + at] = a[1];
    C.ec[at] = a[0];
    C.ec[C.var + at] = a[1];
    halo_put(C, C0, row, at, a[0]);
    halo_put(C, C1, row, at, a[1]);
    halo_put(C, D0, row, at, a[0]);
    halo_put(C, D1, row, at, a[1]);
    C.pb[in] = a[2];
    C.g[in] = a[3];
    C.g[C.ivar + in] = a[4];
  }
}

// The coarsest level, smoothed in FP64 arithmetic (FP32 storage).  Values are
// widened by bit operations, which leave the FP64 unit to the arithmetic: a
// warp's FP64 instruction takes 64 cycles and more, however few of its lanes
// work.  LANES = 2 gives the two variables of a pair to two lanes, so that
// each instruction does both variables' half of the 2x2 system: 19
// instructions a sweep for 30 (2 x 2 cells: 3300 -> 2000 cycles a sweep),
// while all the pairs' lanes fit one warp per scheduler (kCoarsePairs2 pairs);
// more pairs than that take a lane each.
template <int DIM, int LANES, typename F>
__device__ __forceinline__ void cyc_coarsest(const Cyc& A, int x, const Slab& S, bool down, bool emit, int t,
                                             F&& sync) {
  const CycLev& L = A.L[x];
  const int units = (S.n0 >> 1) * (DIM == 3 ? S.n1 : 1) * S.nr;
  const int u = LANES == 2 ? t >> 1 : t;
  const int v = LANES == 2 ? t & 1 : 0;  // this lane's variable
  const bool on = u < units;
  constexpr int NV = 3 - LANES;  // variables a lane holds
  float* const E0 = S.e + v * S.var;
  Pair p;
  float e[2][NV], pb[2];
  float g[2][NV];  // LANES 2: the other variable's right-hand side, which takes this variable's neighbours
  HaloOut H[NV];
#pragma unroll
  for (int w = 0; w < NV; w++) H[w] = halo_out(S, E0 + w * S.var);
  p = pair_of<DIM>(S, L, on ? u : 0);
  const float kc = DIM == 2 ? 4.0f : 6.0f;
#pragma unroll
  for (int b = 0; b < 2; b++) {
#pragma unroll
    for (int w = 0; w < NV; w++) {
      e[b][w] = E0[w * S.var + p.at + b];
      g[b][w] = S.g[(LANES == 2 ? 1 - v : w) * S.ivar + p.in + b];
    }
    pb[b] = S.pb[p.in + b];
  }
  auto partner = [](float q) { return __shfl_xor_sync(0xffffffffu, q, 1); };
  if (down) {
#pragma unroll
    for (int b = 0; b < 2; b++) {
      if (LANES == 1) {
        const float xx = e[b][0], y = e[b][NV - 1];
        const float s0 = pair_sum<DIM, float>(E0, p, b, e[1 - b][0]);
        const float s1 = pair_sum<DIM, float>(E0 + S.var, p, b, e[1 - b][NV - 1]);
        g[b][0] += xx - L.c0 * (s1 - kc * y);
        g[b][NV - 1] += y - xx * (3.0f * pb[b] * (pb[b] + xx) + xx * xx) + L.c1 * (s0 - kc * xx);
      } else {
        const float other = partner(e[b][0]), xx = v ? other : e[b][0], y = v ? e[b][0] : other;
        const float s = pair_sum<DIM, float>(E0, p, b, e[1 - b][0]);
        if (v) g[b][0] += xx - L.c0 * (s - kc * y);
        else g[b][0] += y - xx * (3.0f * pb[b] * (pb[b] + xx) + xx * xx) + L.c1 * (s - kc * xx);
      }
    }
    sync();
  }
  for (int s = 0; s < 2 * A.nsmooth; s++) {
    const int b = p.b0 ^ (s & 1);
    auto dsum = [&](const float* a, float other) {
      const float* c = a + p.at + b;
      double q = f2d(b ? c[p.xr] : c[p.xl]) + f2d(other);
      if (DIM == 2) return q + f2d(c[p.rm]) + f2d(c[p.rp]);
      q = q + f2d(c[p.ym]) + f2d(c[p.yp]);
      return q + (f2d(c[p.rm]) + f2d(c[p.rp]));
    };
    const double pbd = f2d(b ? pb[1] : pb[0]);
    float r[NV];
    if (LANES == 1) {
      const double s0 = dsum(E0, b ? e[0][0] : e[1][0]), s1 = dsum(E0 + S.var, b ? e[0][NV - 1] : e[1][NV - 1]);
      const double xv = f2d(b ? e[1][0] : e[0][0]);
      const double w = pbd + xv;
      const double a21 = -3.0 * w * w - A.cd[2];
      const double b1 = f2d(b ? g[1][0] : g[0][0]) + A.cd[0] * s1;
      const double b2 = f2d(b ? g[1][NV - 1] : g[0][NV - 1]) - A.cd[1] * s0 - xv * xv * (3.0 * pbd + 2.0 * xv);
      const double rdet = __drcp_rn(1.0 - A.cd[3] * a21);
      r[0] = (float)((b1 - A.cd[3] * b2) * rdet);
      r[NV - 1] = (float)((b2 - a21 * b1) * rdet);
    } else {  // the same values, lane 0 | lane 1
      auto swap = [](double q) { return __shfl_xor_sync(0xffffffffu, q, 1); };
      const float own = b ? e[1][0] : e[0][0];
      const float other = partner(own);
      const double xv = f2d(v ? other : own);
      const double sum = dsum(E0, b ? e[0][0] : e[1][0]);
      const double f = __fma_rn(v ? A.cd[0] : -A.cd[1], sum, f2d(b ? g[1][0] : g[0][0]));  // g1 - c1 s0 | b1
      const double f_ = swap(f);
      const double w = (v ? xv : pbd) + xv;                                  // pb + x | 2 x
      const double h = __fma_rn(v ? 3.0 : -3.0, v ? pbd : w, v ? w : 0.0);    // -3 w | 3 pb + 2 x
      const double k = __fma_rn(v ? xv : h, v ? xv : w, v ? 0.0 : -A.cd[2]);  // a21 | x^2
      const double k_ = swap(k);
      const double m = __fma_rn(v ? -k : -A.cd[3], v ? h : k, v ? f_ : 1.0);  // det | b2
      const double m_ = swap(m);
      const double rdet = __drcp_rn(v ? m_ : m);
      // b1 - a12 b2 | b2 - a21 b1
      r[0] = (float)(__fma_rn(v ? -k_ : -A.cd[3], v ? f : m_, v ? m : f_) * rdet);
    }
    if (on)
#pragma unroll
      for (int w = 0; w < NV; w++) {
        if (b) e[1][w] = r[w];
        else e[0][w] = r[w];
        E0[w * S.var + p.at + b] = r[w];
        halo_put(S, H[w], p.row, p.at + b, r[w]);
      }
    if (s + 1 < 2 * A.nsmooth) sync();
  }
  if (emit && on)
#pragma unroll
    for (int w = 0; w < NV; w++) {
      float* const C0 = S.ec + (v + w) * S.var;
      const HaloOut C = halo_out(S, C0);
#pragma unroll
      for (int b = 0; b < 2; b++) {
        const float d = e[b][w] - C0[p.at + b];
        C0[p.at + b] = d;
        halo_put(S, C, p.row, p.at + b, d);
      }
    }
}

// The levels of A once down and up, from the top level's e, g and pb in
// shared memory; the top level's e is final, and every CTA of it past its
// last barrier, at the end.  A level is worked on by as many warps as its
// pairs fill: the others wait for the next level that needs them, so that the
// chain of sweeps through the small levels has the schedulers to itself.
template <int DIM>
__device__ __forceinline__ void cyc_vcycle(const Cyc& A, const SlabInfo* info, int rank, int t, int nt) {
  auto workers = [&](int x) { return info[x].workers; };
  auto smooth = [&](int x, int begin, bool restrict_, bool emit) {
    const bool shared = info[x].shared != 0;
    const int nw = workers(x);
    // barriers of the level's warps, an id a level; shared levels meet across the cluster
    auto local = [&] { asm volatile("bar.sync %0, %1;" ::"r"(1 + x), "r"(nw) : "memory"); };
    auto sync = [&] {
      if (shared) uni::cluster_sync();
      else local();
    };
    // (a shared level) the cluster's barriers count every warp of every CTA
    if (t >= nw || (shared && info[x].own != rank)) {
      const int n = (begin != kTop) + max(0, 2 * A.nsmooth - (restrict_ ? 0 : 1));
      for (int k = 0; k < n; k++) uni::cluster_sync();
    } else {
      const Slab S = slab<DIM, false>(info, x, rank);
      const Slab C = x + 1 < A.nl ? slab<DIM, true>(info, x + 1, rank) : S;
      const int units = (S.n0 >> 1) * (DIM == 3 ? S.n1 : 1) * info[x].maxr;
      if (x == A.nl - 1) {
        if (units <= kCoarsePairs2 && nw >= 2 * units) cyc_coarsest<DIM, 2>(A, x, S, begin == kDown, emit, t, sync);
        else cyc_coarsest<DIM, 1>(A, x, S, begin == kDown, emit, t, sync);
      } else if (units <= nw) {
        cyc_smooth<DIM, 1>(A, x, S, C, begin, restrict_, emit, t, nw, sync, local);
      } else {
        cyc_smooth<DIM, kCycPairs>(A, x, S, C, begin, restrict_, emit, t, nw, sync, local);
      }
    }
    if (shared) uni::cluster_sync();  // what the next level reads has been written
  };
  auto meet = [&](int x) {  // the warps of a level that CTA 0 holds alone
    asm volatile("bar.sync %0, %1;" ::"r"(1 + x), "r"(workers(x)) : "memory");
  };
  for (int x = 0; x < A.nl; x++) {
    const bool shared = info[x].shared != 0;
    if (!shared && (rank || t >= workers(x))) break;
    smooth(x, x ? kDown : kTop, x + 1 < A.nl, x && x + 1 == A.nl);
    if (!shared) meet(x);
  }
  for (int x = A.nl - 2; x >= 0; x--) {
    const bool shared = info[x].shared != 0;
    if (!shared && (rank || t >= workers(x))) continue;
    if (!shared) meet(x);  // the next coarser level is finished
    else if (!info[x + 1].shared) uni::cluster_sync();
    smooth(x, kUp, false, x > 0);
  }
  if (!info[0].shared) __syncthreads();
}

template <int DIM>
__global__ void __launch_bounds__(kCycThreads, 1) k_bx_cycle(float* __restrict__ fp, const __grid_constant__ Cyc A,
                                                             BoxLev T, int fresh) {
  after_previous();
  const int rank = A.ctas > 1 ? uni::my_rank() : 0;
  const int t = threadIdx.x, nt = blockDim.x;
  auto all = [&] {
    if (A.ctas > 1) uni::cluster_sync();
    else __syncthreads();
  };
  __shared__ SlabInfo info[16];
  slab_info<DIM>(A, info, rank, t, nt);
  __syncthreads();
  {  // the top level: e (halo rows too; zero when fresh), g and pb from the colour-split arrays, a pair a thread
    const Slab S = slab<DIM, false>(info, 0, rank);
    const CycLev& L = A.L[0];
    const V2 E = var2(fp, T.oe, T.half), G = var2(fp, T.og, T.half);
    const int pr = (S.n0 >> 1) * (DIM == 3 ? S.n1 : 1);
    if (S.shared || rank == 0)
      for (int u = t; u < pr * (S.nr + 2); u += nt) {
        int r, h, y = 0, k;
        uni::fdivmod(u, L.hx, r, h);
        if (DIM == 3) uni::fdivmod(r, L.d1, k, y);
        else k = r;
        int z = k + S.r0 - 1;
        z = z < 0 ? z + S.N : (z >= S.N ? z - S.N : z);
        const unsigned q = ((unsigned)z * (DIM == 3 ? S.n1 : 1) + y) * T.hh + h;
        const int c = DIM == 3 ? (y + z + 1) & 1 : z & 1;  // colour of cell 2h
        const unsigned i0 = q + (c ? (unsigned)T.half : 0u), i1 = q + (c ? 0u : (unsigned)T.half);
        const int at = k * S.plane + (DIM == 3 ? y * S.n0 : 0) + 2 * h;
        float v[4] = {0.f, 0.f, 0.f, 0.f};
        if (!fresh) v[0] = E.v0[i0], v[1] = E.v0[i1], v[2] = E.v1[i0], v[3] = E.v1[i1];
        S.e[at] = v[0], S.e[at + 1] = v[1];
        S.e[S.var + at] = v[2], S.e[S.var + at + 1] = v[3];
        if (k >= 1 && k <= S.nr) {
          const int in = at - S.plane;
          S.g[in] = G.v0[i0], S.g[in + 1] = G.v0[i1];
          S.g[S.ivar + in] = G.v1[i0], S.g[S.ivar + in + 1] = G.v1[i1];
          S.pb[in] = fp[T.opb + i0], S.pb[in + 1] = fp[T.opb + i1];
        }
      }
  }
  all();
  cyc_vcycle<DIM>(A, info, rank, t, nt);
  const Slab S = slab<DIM, false>(info, 0, rank);
  const CycLev& L = A.L[0];
  const V2 E = var2(fp, T.oe, T.half);
  if (S.shared || rank == 0)
    for (int u = t; u < (S.n0 >> 1) * (DIM == 3 ? S.n1 : 1) * S.nr; u += nt) {
      const Pair p = pair_of<DIM>(S, L, u);
      int r, h;
      uni::fdivmod(u, L.hx, r, h);
      const unsigned q = ((unsigned)S.r0 * (DIM == 3 ? S.n1 : 1) + r) * T.hh + h;
#pragma unroll
      for (int b = 0; b < 2; b++) {
        const unsigned i = q + ((b ^ p.b0) ? (unsigned)T.half : 0u);
        E.v0[i] = S.e[p.at + b];
        E.v1[i] = S.e[S.var + p.at + b];
      }
    }
  all();  // a CTA's shared memory stays while another may still write a halo
}

// After a cycle on the finest level: tracked residual g <- g - M(e) (M at
// this cycle's base field), its per-CTA sums of squares, then qbar += e as
// double-float.  One row (2D) or two rows (3D) per thread; every load
// precedes every store.  Two rows fit 48 registers without spills, five
// blocks per SM (61 registers at four blocks took 185 us at 256^3, 174 us
// capped).
template <int DIM, int R = 1>
__global__ void __launch_bounds__(256, R == 1 ? 6 : 5) k_bx_track_update(float* __restrict__ fp, BoxLev L,
                                                                       long long oqlo, double* __restrict__ partial) {
  after_previous();
  // R rows per thread (y = R yp .. R yp + R - 1): every load of the R cells
  // is issued before the first store, R times the loads in flight
  int x = blockIdx.x * blockDim.x + threadIdx.x;
  int yp = blockIdx.y * blockDim.y + threadIdx.y;
  int z = blockIdx.z;
  float s0 = 0.f, s1 = 0.f;
  if (x < L.n[0] && R * yp < L.n[1]) {
    V2 E = var2(fp, L.oe, L.half), G = var2(fp, L.og, L.half);
    V2 QH = var2(fp, L.opb, L.half), QL = var2(fp, oqlo, L.half);  // the base field is qhi(phi)
    unsigned own[R];
    float a0[R], a1[R], th0[R], tl0[R], th1[R], tl1[R];
    for (int k = 0; k < R; k++) {
      Loc<DIM> l(L, x, R * yp + k, z);
      unsigned i = l.own;
      own[k] = i;
      float h0 = QH.v0[i], h1 = QH.v1[i], lo0 = QL.v0[i], lo1 = QL.v1[i];
      float e0 = E.v0[i], e1 = E.v1[i];
      float m0, m1;
      mop_track<DIM>(E, L, l, h0, m0, m1);
      a0[k] = G.v0[i] - m0;
      a1[k] = G.v1[i] - m1;
      DF t0 = two_sum(h0, e0);
      t0 = fast_two_sum(t0.h, t0.l + lo0);
      DF t1 = two_sum(h1, e1);
      t1 = fast_two_sum(t1.h, t1.l + lo1);
      th0[k] = t0.h, tl0[k] = t0.l, th1[k] = t1.h, tl1[k] = t1.l;
    }
    for (int k = 0; k < R; k++) {
      unsigned i = own[k];
      G.v0[i] = a0[k];
      G.v1[i] = a1[k];
      QH.v0[i] = th0[k];
      QL.v0[i] = tl0[k];
      QH.v1[i] = th1[k];
      QL.v1[i] = tl1[k];
      s0 += a0[k] * a0[k];
      s1 += a1[k] * a1[k];
    }
  }
  cta_sum2(s0, s1, partial);
}

// The true residual r = f - N(qbar) at a cell of the finest level in
// double-float (ErrorAFAS, afasroutines.f90:113-233, with f = (phi_old,
// -phi_old))
template <int DIM>
__device__ __forceinline__ void resid_at(const float* fp, const BoxLev& L, long long oqlo, long long ofhi,
                                         long long oflo, const Loc<DIM>& l, float& a0, float& a1) {
  const DF c0 = {L.c0h, L.c0l}, c1 = {L.c1h, L.c1l};
  const float* QH[2] = {fp + L.opb, fp + L.opb + 2 * L.half};
  const float* QL[2] = {fp + oqlo, fp + oqlo + 2 * L.half};
  const unsigned nbi[6] = {l.xm, l.xp, l.ym, l.yp, l.zm, l.zp};
  DF v[2], nb[2][6];
  for (int q = 0; q < 2; q++) {
    v[q] = {QH[q][l.own], QL[q][l.own]};
    for (int m = 0; m < 2 * DIM; m++) nb[q][m] = {QH[q][nbi[m]], QL[q][nbi[m]]};
  }
  DF f1 = {fp[ofhi + l.own], fp[oflo + l.own]};
  DF lphi = df_lap<DIM>(nb[0], v[0]);
  DF lmu = df_lap<DIM>(nb[1], v[1]);
  // r1 = f1 - (phi - c0 lap(mu)); r2 = -f1 - (mu - phi^3 + c1 lap(phi))
  DF r1 = df_add(df_add(f1, df_neg(v[0])), df_mul(c0, lmu));
  DF p3 = df_mul(df_mul(v[0], v[0]), v[0]);
  DF r2 = df_add(df_add(df_neg(df_add(f1, v[1])), p3), df_neg(df_mul(c1, lphi)));
  a0 = r1.h + r1.l;
  a1 = r2.h + r2.l;
}

// the residual over the level: g is set to it, the per-CTA sums of its
// squares go to partial
template <int DIM>
__global__ void __launch_bounds__(256) k_bx_resid(float* __restrict__ fp, BoxLev L, long long oqlo, long long ofhi,
                                                  long long oflo, double* __restrict__ partial) {
  after_previous();
  int x = blockIdx.x * blockDim.x + threadIdx.x;
  int y = blockIdx.y * blockDim.y + threadIdx.y;
  int z = blockIdx.z;
  float s0 = 0.f, s1 = 0.f;
  if (x < L.n[0] && y < L.n[1]) {
    V2 G = var2(fp, L.og, L.half);
    Loc<DIM> l(L, x, y, z);
    float a0, a1;
    resid_at<DIM>(fp, L, oqlo, ofhi, oflo, l, a0, a1);
    G.v0[l.own] = a0;
    G.v1[l.own] = a1;
    s0 = a0 * a0;
    s1 = a1 * a1;
  }
  cta_sum2(s0, s1, partial);
}

// FP64 q (ghosted Fortran layout) -> qhi/qlo, and f = (phi_old, -phi_old) as
// fhi/flo, on the finest level; two cells (x = 2h, 2h+1) per thread
template <int DIM>
__global__ void __launch_bounds__(256) k_bx_split(const double* __restrict__ pool, long long oq, long long oqold,
                                                  long long sq, int qn0, int qn1, float* __restrict__ fp, BoxLev L,
                                                  long long oqlo, long long ofhi, long long oflo) {
  after_previous();
  int h = blockIdx.x * blockDim.x + threadIdx.x;
  int y = blockIdx.y * blockDim.y + threadIdx.y;
  int z = blockIdx.z;
  if (h >= L.hh || y >= L.n[1]) return;
  long long g = (2 * h + 1) + (long long)(y + 1) * qn0 + (DIM == 3 ? (long long)(z + 1) * qn0 * qn1 : 0);
  double in[2][3];  // the two cells' phi, mu, phi_old, loaded before any store
  for (int b = 0; b < 2; b++) {
    in[b][0] = pool[oq + g + b];
    in[b][1] = pool[oq + sq + g + b];
    in[b][2] = pool[oqold + g + b];
  }
  V2 QH = var2(fp, L.opb, L.half), QL = var2(fp, oqlo, L.half);
  for (int b = 0; b < 2; b++) {
    Loc<DIM> l(L, 2 * h + b, y, z);
    DF s0 = split64(in[b][0]), s1 = split64(in[b][1]), f = split64(in[b][2]);
    QH.v0[l.own] = s0.h;
    QL.v0[l.own] = s0.l;
    QH.v1[l.own] = s1.h;
    QL.v1[l.own] = s1.l;
    fp[ofhi + l.own] = f.h;
    fp[oflo + l.own] = f.l;
  }
}

// k_bx_split for a step that follows a box solve on the same q: with g the
// true residual r_old = f_old - N(q) and f_old in fhi/flo, the residual for
// the new f = (phi_old, -phi_old) is r_old + (f_new - f_old), so g becomes
// g + (d, -d) with d = f_new - f_old in double-float, and the per-CTA sums
// of g^2 go to partial (what k_bx_resid would give, without its
// double-float operator evaluation).
template <int DIM>
__global__ void __launch_bounds__(256) k_bx_split_warm(const double* __restrict__ pool, long long oq, long long oqold,
                                                       long long sq, int qn0, int qn1, float* __restrict__ fp,
                                                       BoxLev L, long long oqlo, long long ofhi, long long oflo,
                                                       double* __restrict__ partial) {
  after_previous();
  int h = blockIdx.x * blockDim.x + threadIdx.x;
  int y = blockIdx.y * blockDim.y + threadIdx.y;
  int z = blockIdx.z;
  float s0 = 0.f, s1 = 0.f;
  if (h < L.hh && y < L.n[1]) {
    long long g = (2 * h + 1) + (long long)(y + 1) * qn0 + (DIM == 3 ? (long long)(z + 1) * qn0 * qn1 : 0);
    V2 QH = var2(fp, L.opb, L.half), QL = var2(fp, oqlo, L.half), G = var2(fp, L.og, L.half);
    double in[2][3];
    unsigned own[2];
    float fo[2][2], go[2][2];  // old f (hi, lo) and g, loaded before any store
    for (int b = 0; b < 2; b++) {
      in[b][0] = pool[oq + g + b];
      in[b][1] = pool[oq + sq + g + b];
      in[b][2] = pool[oqold + g + b];
      Loc<DIM> l(L, 2 * h + b, y, z);
      own[b] = l.own;
      fo[b][0] = fp[ofhi + l.own];
      fo[b][1] = fp[oflo + l.own];
      go[b][0] = G.v0[l.own];
      go[b][1] = G.v1[l.own];
    }
    for (int b = 0; b < 2; b++) {
      unsigned i = own[b];
      DF s0v = split64(in[b][0]), s1v = split64(in[b][1]), f = split64(in[b][2]);
      DF d = df_add(f, df_neg(DF{fo[b][0], fo[b][1]}));
      DF r1 = df_add(DF{go[b][0], 0.f}, d), r2 = df_add(DF{go[b][1], 0.f}, df_neg(d));
      float a0 = r1.h + r1.l, a1 = r2.h + r2.l;
      QH.v0[i] = s0v.h;
      QL.v0[i] = s0v.l;
      QH.v1[i] = s1v.h;
      QL.v1[i] = s1v.l;
      fp[ofhi + i] = f.h;
      fp[oflo + i] = f.l;
      G.v0[i] = a0;
      G.v1[i] = a1;
      s0 += a0 * a0;
      s1 += a1 * a1;
    }
  }
  cta_sum2(s0, s1, partial);
}

// qhi + qlo -> FP64 q (interior of the finest level)
template <int DIM>
__global__ void __launch_bounds__(256) k_bx_merge(double* __restrict__ pool, long long oq, long long sq, int qn0,
                                                  int qn1, float* __restrict__ fp, BoxLev L, long long oqlo) {
  after_previous();
  int h = blockIdx.x * blockDim.x + threadIdx.x;
  int y = blockIdx.y * blockDim.y + threadIdx.y;
  int z = blockIdx.z;
  if (h >= L.hh || y >= L.n[1]) return;
  long long g = (2 * h + 1) + (long long)(y + 1) * qn0 + (DIM == 3 ? (long long)(z + 1) * qn0 * qn1 : 0);
  V2 QH = var2(fp, L.opb, L.half), QL = var2(fp, oqlo, L.half);
  float hi[2][2], lo[2][2];  // loaded before any store
  for (int b = 0; b < 2; b++) {
    Loc<DIM> l(L, 2 * h + b, y, z);
    hi[b][0] = QH.v0[l.own];
    hi[b][1] = QH.v1[l.own];
    lo[b][0] = QL.v0[l.own];
    lo[b][1] = QL.v1[l.own];
  }
  for (int b = 0; b < 2; b++)
    for (int v = 0; v < 2; v++) pool[oq + v * sq + g + b] = f2d(hi[b][v]) + f2d(lo[b][v]);
}

// ---------------------------------------------------------------------------
// The whole solve of a box whose finest level fits the cluster (k_bx_cycle)
// as one launch: the split of q, the starting residual, the V-cycles, the
// tracked residual and qbar += e after each, the confirming residuals, the
// exit test of box_iterations and the write-back of q with its periodic
// images.  e, g and pb stay in shared memory from cycle to cycle; qhi, qlo
// and f stay where the other kernels keep them (a cluster barrier makes one
// CTA's writes visible to the others).  Per cell it computes what the
// separate kernels compute; the norms add the same squares in another order,
// in FP32 over a warp's cells (at most 128; there a CTA's 256 or 512) and in
// FP64 from there.
//
// A step of such a box was some 14 launches and a graph with a conditional
// loop of six launches a V-cycle; now it is this one, the fill of the coarse
// levels and one wait.  A step of five V-cycles at 32^2: 285 -> 200 us; of
// seven at 128^2: 510 -> 440 us.  What bounds it is the chain of sweeps.
constexpr int kSolveMaxCycles = 64;
struct BoxSolve {
  long long oqlo, ofhi, oflo;      // float offsets
  long long oq, oqold, sq;         // FP64 pool: q, qold (cell (0,0,0) of variable 1), variable stride
  int qn0, qn1;
  double tol, count;               // exit tolerance, ErrorAFAS denominator
  int maxv, errortype, warm;
};
// what the host reads (pinned memory)
struct BoxSolveOut {
  int it, conv, status, nconfirm;
  double res[kSolveMaxCycles];
};

template <int DIM>
__global__ void __launch_bounds__(kCycThreads, 1) k_bx_solve(float* __restrict__ fp, double* __restrict__ pool,
                                                             const __grid_constant__ Cyc A, BoxLev T, BoxSolve B,
                                                             BoxSolveOut* __restrict__ out) {
  after_previous();
  const int rank = A.ctas > 1 ? uni::my_rank() : 0;
  const int t = threadIdx.x, nt = blockDim.x;
  static_assert(kCycThreads <= 16 * 32, "a half-warp adds the sums of the warps");
  __shared__ float wsum[2][kCycThreads / 32];
  __shared__ double part[2][32];  // two norms' worth: a CTA may start the next while another still adds up this one
  __shared__ double norm_now;
  __shared__ int verdict;
  int turn = 0;
  auto all = [&] {
    if (A.ctas > 1) uni::cluster_sync();
    else __syncthreads();
  };
  __shared__ SlabInfo info[16];
  slab_info<DIM>(A, info, rank, t, nt);
  __syncthreads();
  const Slab S = slab<DIM, false>(info, 0, rank);
  const CycLev& L = A.L[0];
  const int n1 = DIM == 3 ? S.n1 : 1;
  // a top level that CTA 0 holds alone leaves the others without cells
  const int units = S.shared || rank == 0 ? (S.n0 >> 1) * n1 * S.nr : 0;
  const V2 G = var2(fp, T.og, T.half), QH = var2(fp, T.opb, T.half), QL = var2(fp, B.oqlo, T.half);
  // pair u's global y, z and the element of its cell b in a colour-split array
  struct At {
    int x, y, z;
    unsigned i[2];
  };
  auto at = [&](int u, const Pair& p) {
    At a;
    int r, h;
    uni::fdivmod(u, L.hx, r, h);
    a.x = 2 * h;
    if (DIM == 3) {
      int k;
      uni::fdivmod(r, L.d1, k, a.y);
      a.z = k + S.r0;
    } else {
      a.y = r + S.r0;
      a.z = 0;
    }
    const unsigned q = ((unsigned)S.r0 * n1 + r) * T.hh + h;
    for (int b = 0; b < 2; b++) a.i[b] = q + ((b ^ p.b0) ? (unsigned)T.half : 0u);
    return a;
  };
  auto fp64_at = [&](const At& a) {  // offset of cell (x, y, z) in a ghosted plane of q
    return (long long)(a.x + 1) + (long long)(a.y + 1) * B.qn0 +
           (DIM == 3 ? (long long)(a.z + 1) * B.qn0 * B.qn1 : 0);
  };
  // ErrorAFAS of the squares each thread summed, in every CTA, and what
  // judge(it) makes of it: by one thread, an FP64 comparison of every warp
  // would take the FP64 unit longer than the norm itself
  auto norm = [&](float s0, float s1, auto&& judge) {
    for (int o = 16; o > 0; o >>= 1) {
      s0 += __shfl_down_sync(0xffffffffu, s0, o);
      s1 += __shfl_down_sync(0xffffffffu, s1, o);
    }
    if ((t & 31) == 0) wsum[0][t >> 5] = s0, wsum[1][t >> 5] = s1;
    double* const sums = part[turn];
    turn ^= 1;
    __syncthreads();
    if (t < 32) {
      // in FP64 from a warp's cells on, half a warp a variable; the warps
      // without a pair hold zeros, whose additions are left out
      const int warps = (units + 31) >> 5;
      double s = f2d((t & 15) < nt / 32 ? wsum[t >> 4][t & 15] : 0.f);
      for (int o = 8; o > 0; o >>= 1)
        if (o < warps) s += __shfl_down_sync(0xffffffffu, s, o, 16);
      const double a = __shfl_sync(0xffffffffu, s, 0), b = __shfl_sync(0xffffffffu, s, 16);
      if (t < A.ctas) {  // to every CTA
        double* p = A.ctas > 1 ? uni::on_rank(sums, t) : sums;
        p[rank] = a;
        p[16 + rank] = b;
      }
    }
    all();
    if (t < 32) {
      double a = t < A.ctas ? sums[t] : 0.0, b = t < A.ctas ? sums[16 + t] : 0.0;
      for (int o = 8; o > 0; o >>= 1)
        if (o < A.ctas) {
          a += __shfl_down_sync(0xffffffffu, a, o);
          b += __shfl_down_sync(0xffffffffu, b, o);
        }
      if (t == 0) {
        if (B.errortype == 1) {
          norm_now = sqrt((a + b) / B.count);
        } else {
          const double r0 = sqrt(a / (0.5 * B.count)), r1 = sqrt(b / (0.5 * B.count));
          norm_now = r1 > r0 ? r1 : r0;
        }
        verdict = judge(norm_now);
      }
    }
    __syncthreads();
    return verdict;
  };
  // the true residual to g; its norm
  auto confirm = [&](auto&& judge) {
    float s0 = 0.f, s1 = 0.f;
    for (int u = t; u < units; u += nt) {
      const Pair p = pair_of<DIM>(S, L, u);
      const At a = at(u, p);
#pragma unroll 1
      for (int b = 0; b < 2; b++) {
        const Loc<DIM> l(T, a.x + b, a.y, a.z);
        float r0, r1;
        resid_at<DIM>(fp, T, B.oqlo, B.ofhi, B.oflo, l, r0, r1);
        S.g[p.in + b] = r0;
        S.g[S.ivar + p.in + b] = r1;
        s0 += r0 * r0;
        s1 += r1 * r1;
      }
    }
    return norm(s0, s1, judge);
  };
  // q and qold split into float pairs (k_bx_split, k_bx_split_warm)
  float w0 = 0.f, w1 = 0.f;
  for (int u = t; u < units; u += nt) {
    const Pair p = pair_of<DIM>(S, L, u);
    const At a = at(u, p);
    const long long g = fp64_at(a);
#pragma unroll
    for (int b = 0; b < 2; b++) {
      const unsigned i = a.i[b];
      const DF s0 = split64(pool[B.oq + g + b]), s1 = split64(pool[B.oq + B.sq + g + b]);
      const DF f = split64(pool[B.oqold + g + b]);
      if (B.warm) {
        const DF d = df_add(f, df_neg(DF{fp[B.ofhi + i], fp[B.oflo + i]}));
        const DF r1 = df_add(DF{G.v0[i], 0.f}, d), r2 = df_add(DF{G.v1[i], 0.f}, df_neg(d));
        const float a0 = r1.h + r1.l, a1 = r2.h + r2.l;
        S.g[p.in + b] = a0;
        S.g[S.ivar + p.in + b] = a1;
        w0 += a0 * a0;
        w1 += a1 * a1;
      }
      QH.v0[i] = s0.h;
      QL.v0[i] = s0.l;
      QH.v1[i] = s1.h;
      QL.v1[i] = s1.l;
      fp[B.ofhi + i] = f.h;
      fp[B.oflo + i] = f.l;
      S.pb[p.in + b] = s0.h;
    }
  }
  auto clear = [&] {  // e = 0, halo rows too
    if (units)
      for (int q = t; q < 2 * S.var; q += nt) S.e[q] = 0.f;
  };
  clear();
  all();
  double r_sync = 0.0;  // the last true residual (thread 0)
  enum { kNonfinite = 1, kConfirm = 2, kConverged = 4 };
  auto judge_true = [&](double r) {
    r_sync = r;
    return !isfinite(r) ? kNonfinite : (r < B.tol ? kConverged : 0);
  };
  int status = (B.warm ? norm(w0, w1, judge_true) : confirm(judge_true)) & kNonfinite, conv = 0, it = 0, nconfirm = 0;
  while (!status && it < B.maxv) {
    it++;
    cyc_vcycle<DIM>(A, info, rank, t, nt);
    // g -= M(e), then qbar += e (k_bx_track_update)
    float s0 = 0.f, s1 = 0.f;
    for (int u = t; u < units; u += nt) {
      const Pair p = pair_of<DIM>(S, L, u);
      const At a = at(u, p);
#pragma unroll
      for (int b = 0; b < 2; b++) {
        const float *E0 = S.e + p.at + b, *E1 = E0 + S.var;
        const float x = E0[0], y = E1[0], pb = S.pb[p.in + b];
        auto diff = [&](const float* c, float v) {  // ndiff
          const float q = (c[b ? -1 : p.xl] - v) + (c[b ? p.xr : 1] - v);
          if (DIM == 2) return q + ((c[p.rm] - v) + (c[p.rp] - v));
          float z = q + ((c[p.ym] - v) + (c[p.yp] - v));
          z += (c[p.rm] - v) + (c[p.rp] - v);
          return z;
        };
        const float m0 = x - L.c0 * diff(E1, y);
        const float m1 = y - x * (3.0f * pb * (pb + x) + x * x) + L.c1 * diff(E0, x);
        const float a0 = S.g[p.in + b] - m0, a1 = S.g[S.ivar + p.in + b] - m1;
        const unsigned i = a.i[b];
        DF t0 = two_sum(pb, x);
        t0 = fast_two_sum(t0.h, t0.l + QL.v0[i]);
        DF t1 = two_sum(QH.v1[i], y);
        t1 = fast_two_sum(t1.h, t1.l + QL.v1[i]);
        S.g[p.in + b] = a0;
        S.g[S.ivar + p.in + b] = a1;
        S.pb[p.in + b] = t0.h;
        QH.v0[i] = t0.h;
        QL.v0[i] = t0.l;
        QH.v1[i] = t1.h;
        QL.v1[i] = t1.l;
        s0 += a0 * a0;
        s1 += a1 * a1;
      }
    }
    int v = norm(s0, s1, [&](double r) {
      return !isfinite(r) ? kNonfinite : (r < B.tol || r < 1e-5 * r_sync || it >= B.maxv ? kConfirm : 0);
    });
    clear();  // after norm's barrier: every read of e is done
    if (v & kConfirm) {
      v = confirm(judge_true);
      nconfirm++;
    }
    status = v & kNonfinite;
    conv = v & kConverged;
    if (rank == 0 && t == 0 && !status) out->res[it - 1] = norm_now;
    if (conv) break;
    all();  // e is zero in every CTA
  }
  // q, its periodic images, and the residual the next step starts from
  for (int u = t; u < units; u += nt) {
    const Pair p = pair_of<DIM>(S, L, u);
    const At a = at(u, p);
    const long long g = fp64_at(a);
#pragma unroll
    for (int b = 0; b < 2; b++) {
      const unsigned i = a.i[b];
      G.v0[i] = S.g[p.in + b];
      G.v1[i] = S.g[S.ivar + p.in + b];
      const double v[2] = {f2d(QH.v0[i]) + f2d(QL.v0[i]), f2d(QH.v1[i]) + f2d(QL.v1[i])};
      const int x = a.x + b;
      const long long dx = x == 0 ? T.n[0] : (x == T.n[0] - 1 ? -T.n[0] : 0);
      const long long dy = (a.y == 0 ? T.n[1] : (a.y == T.n[1] - 1 ? -T.n[1] : 0)) * (long long)B.qn0;
      const long long dz =
          DIM == 3 ? (a.z == 0 ? T.n[2] : (a.z == T.n[2] - 1 ? -T.n[2] : 0)) * (long long)B.qn0 * B.qn1 : 0;
#pragma unroll
      for (int m = 0; m < (1 << DIM); m++) {
        if (((m & 1) && !dx) || ((m & 2) && !dy) || ((m & 4) && !dz)) continue;
        const long long o = g + b + (m & 1 ? dx : 0) + (m & 2 ? dy : 0) + (m & 4 ? dz : 0);
        pool[B.oq + o] = v[0];
        pool[B.oq + B.sq + o] = v[1];
      }
    }
  }
  if (rank == 0 && t == 0) {
    out->it = it;
    out->conv = conv != 0;
    out->status = status != 0;
    out->nconfirm = nconfirm;
  }
  all();  // a CTA's shared memory stays while another may still address it
}

// ---------------------------------------------------------------------------
// host side

struct Launch {
  dim3 g, b;
};
// threads over (nx, ny, nz) with up to 128 along x and 256 per block
Launch shape(int nx, int ny, int nz) {
  int tx = nx >= 128 ? 128 : nx;
  int ty = std::max(1, 256 / tx);
  if (ty > ny) ty = ny;
  return {dim3((nx + tx - 1) / tx, (ny + ty - 1) / ty, nz), dim3(tx, ty, 1)};
}
long long ctas(const Launch& s) { return (long long)s.g.x * s.g.y * s.g.z; }

#define BX_LAUNCH(H, SH, KER, ...)                                            \
  do {                                                                        \
    if ((H).ndims == 2) launch_after(KER<2>, (SH).g, (SH).b, 0, (H).s, __VA_ARGS__);    \
    else launch_after(KER<3>, (SH).g, (SH).b, 0, (H).s, __VA_ARGS__);                   \
    int r__ = after_launch(H, 1);                                             \
    if (r__) return r__;                                                      \
  } while (0)

BoxLev& B(Hier& H, int level) { return H.blev[level + kMaxDepth]; }

// The staged sweep (box_sweep 2) applies to 3D levels whose rows are whole
// 16-byte units and whose planes split into whole 8-row tiles, large enough
// to fill the GPU; two stages of 8 rows measured fastest of the staged forms.
constexpr int kTileT = 8, kTileNS = 2;
bool staged_relax(const Hier& H, const BoxLev& L) {
  if (H.box_sweep != 2 || H.ndims != 3) return false;
  long long smem = (long long)kTileNS * tile_stage_floats(kTileT, L.hh) * 4;
  return L.hh % 4 == 0 && L.hh >= 64 && smem <= 200 * 1024 && L.n[1] % kTileT == 0 &&
         (kTileT * L.hh) % kTileThreads == 0;
}

int launch_staged(Hier& H, const BoxLev& L, int c, int first) {
  int occ = 0;
  int smem = kTileNS * tile_stage_floats(kTileT, L.hh) * (int)sizeof(float);
  auto ker = k_bx_relax_tiled<kTileT, kTileNS>;
  cudaError_t e = cudaFuncSetAttribute(ker, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(k_bx_relax_tiled)");
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, ker, kTileThreads, smem);
  if (e != cudaSuccess || occ < 1) return cuda_fail(e, "occupancy(k_bx_relax_tiled)");
  int ntiles = (L.n[1] / kTileT) * L.n[2];
  int grid = std::min(ntiles, occ * H.box_sms);
  launch_after(ker, grid, kTileThreads, smem, H.s, H.fpool, L, c, first);
  return after_launch(H, 1);
}

// The one-pass smoothing (box_sweep 3): 3D levels whose colour rows hold 128
// cells (tiles of 8 rows; the ring fills 224 KB of shared memory), at least
// one tile and its halo per plane.  Levels of 64-cell rows (tiles of 16 rows)
// compile but measured slower than four sweeps on a GB300 (128^3: 62 against
// 36 us, at a time when a level was cut into whole tiles by a quarter of the
// planes, 64 CTAs there; not measured again with smooth_split), so they keep
// the sweeps.
int smooth_rows(const BoxLev& L) {
  const int ty = L.hh == 128 ? 8 : 0;
  return ty && L.n[1] % ty == 0 && L.n[1] >= ty + 2 * kSmStages ? ty : 0;
}
bool smooth_fits(const Hier& H, const BoxLev& L) {
  return H.ndims == 3 && L.n[2] >= kSmStages && smooth_rows(L) > 0;
}

// cuTensorMapEncodeTiled through the runtime's driver entry point (no link
// against the driver library); null when the driver does not provide it
PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
  static const PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      p = nullptr;
    return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  }();
  return fn;
}

// the tensor map of a level's e arrays at offset oe: [array][z][y][h] with
// h innermost, a box of four rows of one array
int e_tensor_map(Hier& H, const BoxLev& L, long long oe, CUtensorMap* m) {
  const PFN_cuTensorMapEncodeTiled_v12000 enc = tensor_map_encoder();
  if (!enc) return cuda_fail(cudaErrorNotSupported, "cuTensorMapEncodeTiled entry point");
  const cuuint64_t dims[4] = {(cuuint64_t)L.hh, (cuuint64_t)L.n[1], (cuuint64_t)L.n[2], 4};
  const cuuint64_t strides[3] = {(cuuint64_t)L.hh * 4, (cuuint64_t)L.hh * L.n[1] * 4, (cuuint64_t)L.half * 4};
  const cuuint32_t box[4] = {(cuuint32_t)L.hh, 4, 1, 1};
  const cuuint32_t es[4] = {1, 1, 1, 1};
  CUresult r = enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, H.fpool + oe, dims, strides, box, es,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return cuda_fail(cudaErrorInvalidValue, "cuTensorMapEncodeTiled");
  return BSAMG_OK;
}

// The split of a level of `tiles` y-tiles of n2 planes over at most `ctas`
// CTAs: a CTA passes over its planes and 2 NS more for every tile it works
// on, so the line is cut by passes, not by planes, into the smallest number
// of passes a CTA that the CTAs suffice for.  Every SM has its share whatever
// the extents (256^3: 150 CTAs of 64 passes, 166 us, instead of 128 CTAs, four
// to a tile, of 72 passes, 182 us).
// A CTA goes on to the next tile only for kSmTail planes or more.
constexpr int kSmTail = 4;
int smooth_split(int tiles, int n2, int ctas, SmoothSplit& S) {
  const int total = tiles * n2;
  auto cut = [&](int passes) {  // the CTAs it takes; more than `ctas` count as one more
    int k = 0;
    for (int p = 0; p < total && k <= ctas; k++) {
      if (k < ctas) S.start[k] = p;
      for (int left = passes; p < total;) {
        const int room = left - 2 * kSmStages, rest = n2 - p % n2;
        if (room < std::min(rest, left == passes ? 1 : kSmTail)) break;
        const int take = std::min(room, rest);
        p += take;
        left -= take + 2 * kSmStages;
      }
    }
    return k;
  };
  int lo = std::min(kSmMinPlanes, n2) + 2 * kSmStages, hi = total + tiles * 2 * kSmStages;
  while (lo < hi) {
    const int mid = (lo + hi) / 2;
    if (cut(mid) <= ctas) hi = mid;
    else lo = mid + 1;
  }
  const int k = cut(lo);
  S.start[k] = total;
  return k;
}

// out_oe = e after two red-black passes from e at in.oe (fresh: from zero)
int bx_smooth(Hier& H, const BoxLev& in, long long out_oe, bool fresh) {
  const int ty = smooth_rows(in);
  SmoothSplit split;
  const int ctas = smooth_split(in.n[1] / ty, in.n[2], std::max(1, std::min(H.box_sms, kSmMaxCtas)), split);
  size_t smem = (size_t)smooth_slots(kSmStages) * smooth_slot_floats(ty, in.hh) * sizeof(float);
  static std::atomic<unsigned long long> attr;  // the kernels' shared-memory limit, per device
  if (needs_setup(attr, H.ctx->device)) {
    for (auto kf : {k_bx_smooth<8, 128, true>, k_bx_smooth<8, 128, false>}) {
      cudaError_t e = cudaFuncSetAttribute(kf, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(k_bx_smooth)");
    }
    mark_setup(attr, H.ctx->device);
  }
  CUtensorMap emap;
  int r = e_tensor_map(H, in, in.oe, &emap);
  if (r) return r;
  auto ker = fresh ? k_bx_smooth<8, 128, true> : k_bx_smooth<8, 128, false>;
  launch_after(ker, ctas, kSmThreads, smem, H.s, H.fpool, in, out_oe, split, emap);
  return after_launch(H, 1);
}
bool smooth_applies(const Hier& H, const BoxLev& L, int nsmooth) {
  return H.box_sweep == 3 && nsmooth == 2 && L.oe2 >= 0;
}

int bx_relax(Hier& H, int level, int c, int first) {
  BoxLev& L = B(H, level);
  if (staged_relax(H, L)) return launch_staged(H, L, c, first);
  if ((H.box_sweep == 1 || H.box_sweep == 3) && H.ndims == 3 && L.n[1] % 4 == 0) {
    // four rows per thread at five blocks per SM (40 registers): four
    // cells' loads in flight per thread
    Launch sh = shape(L.hh, L.n[1] / 4, L.n[2]);
    launch_after(k_bx_relax<3, 4, 5>, sh.g, sh.b, 0, H.s, H.fpool, L, c, first);
    return after_launch(H, 1);
  }
  Launch sh = shape(L.hh, L.n[1] / 2, L.n[2]);
  BX_LAUNCH(H, sh, k_bx_relax, H.fpool, L, c, first);
  return BSAMG_OK;
}

int bx_restrict_load(Hier& H, const BoxLev& F, const BoxLev& C) {
  if (H.ndims == 2) {
    const Launch sh = shape(C.n[0], C.n[1], 1);
    launch_after(k_bx_restrict_load, sh.g, sh.b, 0, H.s, H.fpool, F, C);
    return after_launch(H, 1);
  }
  const int nx = C.n[0] / kRestrictCells, tx = std::min(nx, kRestrictThreads);
  const int ty = std::max(1, std::min(kRestrictThreads / tx, C.n[1]));
  launch_after(k_bx_restrict_rows, dim3((nx + tx - 1) / tx, (C.n[1] + ty - 1) / ty, C.n[2]), dim3(tx, ty), 0, H.s,
               H.fpool, F, C);
  return after_launch(H, 1);
}

// coarse: the V-cycle's coarsest level, smoothed in FP64 arithmetic
int bx_level_relax(Hier& H, int level, int nsmooth, bool fresh, bool coarse = false) {
  for (int pass = 1; pass <= nsmooth; pass++)
    for (int c = 0; c < 2; c++) {
      const int first = (fresh && pass == 1) ? c + 1 : 0;
      if (coarse) {
        BoxLev& L = B(H, level);
        Launch sh = shape(L.hh, L.n[1], L.n[2]);
        BX_LAUNCH(H, sh, k_bx_relax64, H.fpool, L, c, first);
        continue;
      }
      int r = bx_relax(H, level, c, first);
      if (r) return r;
    }
  return BSAMG_OK;
}

// clusters of `ctas` CTAs with smem bytes that fit at once; raises the
// kernel's limits
int cycle_fit(int ndims, int ctas, int smem) {
  auto fit = [&](auto k) {
    if (cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) return 0;
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kUniSmemMax) != cudaSuccess) return 0;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3(kCycThreads);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = ctas;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, k, &cfg) != cudaSuccess) return 0;
    return n;
  };
  const int n = ndims == 2 ? std::min(fit(k_bx_cycle<2>), fit(k_bx_solve<2>))
                           : std::min(fit(k_bx_cycle<3>), fit(k_bx_solve<3>));
  cudaGetLastError();  // a shape that does not fit is an answer, not an error
  return n;
}

// The cluster's plan for the levels top .. minlevel with the first `share`
// of them shared out; false when it does not fit (shared memory, pairs a
// thread, the coarsest level's one pair a thread)
bool cycle_layout(Hier& H, int top, int minlevel, int nsmooth, int share, int base, Cyc& A, int* smem) {
  const int D = H.ndims;
  A = Cyc{};
  A.nl = top - minlevel + 1;
  A.nsmooth = nsmooth;
  A.ctas = 1;
  int nc = 1;
  if (share) {
    // every CTA's rows are whole rows of level `base`: the first level CTA 0
    // holds alone (each CTA restricts whole coarse rows), or the last one when
    // all are shared.  A base above that has one row a CTA, and the shared
    // levels from it down are held by every 2nd, 4th, .. CTA, two rows each.
    nc = B(H, top - base).n[D - 1];
    A.ctas = std::min(16, nc);
    const int folds = std::min(share, A.nl) - base;  // levels held by some CTAs only
    if (A.ctas < 2 || (base < std::min(share, A.nl - 1) && (A.ctas != nc || (A.ctas >> folds) < 2))) return false;
  }
  for (int r = 0; r <= A.ctas; r++) A.row0[r] = r * nc / A.ctas;
  long long o = 0, scratch = 0;
  auto add = [&](long long n) {
    const long long at = o;
    o += (n + 3) & ~3LL;
    return (int)at;
  };
  auto dv = [](int d) { return UniDiv{d, d <= 1 ? 0u : 0xFFFFFFFFu / (unsigned)d + 1u}; };
  for (int x = 0; x < A.nl; x++) {
    const BoxLev& P = B(H, top - x);
    CycLev& L = A.L[x];
    L.n0 = P.n[0], L.n1 = P.n[1], L.N = P.n[D - 1];
    L.mul = x < share ? 1 << std::max(0, base - x) : 0;
    L.down = std::max(0, x - base);
    L.fold = base < std::min(share, A.nl - 1) && x >= base ? 1 + x - base : 0;
    L.maxr = L.N;
    if (L.mul) {
      const int st = 1 << L.fold;
      if (A.ctas % st) return false;
      L.maxr = 0;
      for (int r = 0; r < A.ctas; r += st)
        L.maxr = std::max(L.maxr, ((A.row0[r + st] * L.mul) >> L.down) - ((A.row0[r] * L.mul) >> L.down));
      if (L.maxr < 1) return false;
    }
    const long long plane = (long long)P.n[0] * (D == 3 ? P.n[1] : 1);
    const long long pairs = plane / 2 * L.maxr;
    if (pairs > kCycThreads * (x + 1 < A.nl ? kCycPairs : 1)) return false;
    L.e = add(2 * plane * (L.maxr + 2));
    L.ec = x ? add(2 * plane * (L.maxr + 2)) : 0;
    L.g = add(2 * plane * L.maxr);
    L.pb = add(plane * L.maxr);
    L.c0 = P.c0, L.c1 = P.c1, L.tmp3 = P.tmp3, L.a12 = P.a12;
    L.hx = dv(P.n[0] / 2), L.d1 = dv(P.n[1]), L.hc = dv(P.n[0] / 2), L.dc1 = dv(std::max(1, P.n[1] / 2));
    // the sums of the restriction keep the order of each size of level: small
    // levels colour by colour, the others as k_bx_restrict_load and _rows
    L.by_colour = 2 * P.half <= 8192;
    if (x + 1 < A.nl) scratch = std::max(scratch, 4 * pairs);
    if (o * 4 > kUniSmemMax || A.nl > 15) return false;  // (a named barrier a level)
  }
  A.scratch = add(scratch);
  for (int v = 0; v < 4; v++) A.cd[v] = B(H, minlevel).cd[v];
  *smem = (int)(o * 4);
  return *smem <= kUniSmemMax;
}

// The level from which the V-cycle runs in the cluster (the highest that
// fits, or none), and the split of its levels: the cheapest by a model of a
// sweep -- a barrier of the cluster or of the CTA and the issue slots of
// about 70 instructions a pair.
bool cycle_plan(Hier& H, int level, int minlevel, int nsmooth, Cyc& best, int* smem, int* at) {
  for (int top = level; top >= minlevel; top--) {
    struct Form {
      double us;
      int smem;
      Cyc A;
    };
    std::vector<Form> forms;
    const int nl = top - minlevel + 1;
    for (int share = 0; share <= nl; share++)
      for (int base = std::min(share, nl - 1); base >= std::min(std::min(share, 1), nl - 1); base--) {
        Form f{0.0, 0, {}};
        if (!cycle_layout(H, top, minlevel, nsmooth, share, base, f.A, &f.smem)) continue;
        for (int x = 0; x < f.A.nl; x++) {
          const double pairs = (double)B(H, top - x).half / (x < share ? f.A.ctas >> f.A.L[x].fold : 1);
          f.us += (x < share ? 0.75 : 0.3) + pairs * 70 / 32 / 4 / 2000.0 * 1.5;
        }
        forms.push_back(f);
      }
    std::stable_sort(forms.begin(), forms.end(), [](const Form& a, const Form& b) { return a.us < b.us; });
    for (const Form& f : forms)  // the cheapest that fits: asking the runtime costs tens of microseconds
      if (cycle_fit(H.ndims, f.A.ctas, f.smem) >= 1) {
        best = f.A;
        *smem = f.smem;
        *at = top;
        return true;
      }
  }
  return false;
}

// AFASVcycle (afasroutines.f90:495-529) on the correction
int bx_vcycle_from(Hier& H, int level, int minlevel, int nsmooth, bool fresh, const Cyc& cyc, int cyc_smem, int cyc_at) {
  if (level <= cyc_at) {  // the rest of the V-cycle in one cluster launch
    const BoxLev& T = B(H, level);
    auto k = H.ndims == 2 ? k_bx_cycle<2> : k_bx_cycle<3>;
    cudaError_t e = launch_cluster(k, cyc.ctas, kCycThreads, cyc_smem, H.s, H.fpool, cyc, T, fresh ? 1 : 0);
    if (e != cudaSuccess) return cuda_fail(e, "coarse V-cycle launch");
    return after_launch(H, 1);
  }
  if (level > minlevel && smooth_applies(H, B(H, level), nsmooth)) {
    // one-pass smoothings: e to the level's second array before the
    // coarse correction and back after it
    BoxLev F = B(H, level), Fb = F;
    Fb.oe = F.oe2;
    const BoxLev& C = B(H, level - 1);
    Launch sc = shape(C.n[0], C.n[1], C.n[2]);
    int r = bx_smooth(H, F, F.oe2, fresh);
    if (r) return r;
    if ((r = bx_restrict_load(H, Fb, C))) return r;
    BX_LAUNCH(H, sc, k_bx_coarse_op, H.fpool, C);
    if ((r = bx_vcycle_from(H, level - 1, minlevel, nsmooth, false, cyc, cyc_smem, cyc_at))) return r;
    BX_LAUNCH(H, sc, k_bx_prolong, H.fpool, Fb, C);
    return bx_smooth(H, Fb, F.oe, false);
  }
  int r = bx_level_relax(H, level, nsmooth, fresh, level == minlevel);
  if (r) return r;
  if (level > minlevel) {
    BoxLev &F = B(H, level), &C = B(H, level - 1);
    Launch sc = shape(C.n[0], C.n[1], C.n[2]);
    if ((r = bx_restrict_load(H, F, C))) return r;
    BX_LAUNCH(H, sc, k_bx_coarse_op, H.fpool, C);
    if ((r = bx_vcycle_from(H, level - 1, minlevel, nsmooth, false, cyc, cyc_smem, cyc_at))) return r;
    BX_LAUNCH(H, sc, k_bx_prolong, H.fpool, F, C);
    if ((r = bx_level_relax(H, level, nsmooth, false))) return r;
  }
  return BSAMG_OK;
}

// the plan of the whole V-cycle from the finest level, where that fits: made
// once per (finest, minlevel, nsmooth) and coefficients
bool solve_plan(Hier& H, int finest, int minlevel, int nsmooth, Cyc& cyc, int* smem) {
  auto key = std::make_tuple(finest, minlevel, nsmooth);
  if (!H.box_plan || H.box_plan_key != key) {
    auto pl = std::make_shared<std::pair<Cyc, int>>();
    int at = finest - 1;
    if (!cycle_plan(H, finest, minlevel, nsmooth, pl->first, &pl->second, &at) || at != finest) pl->second = -1;
    H.box_plan = pl;
    H.box_plan_key = key;
  }
  const auto& pl = *std::static_pointer_cast<std::pair<Cyc, int>>(H.box_plan);
  if (pl.second < 0) return false;
  cyc = pl.first;
  *smem = pl.second;
  return true;
}

int bx_vcycle(Hier& H, int level, int minlevel, int nsmooth, bool fresh) {
  Cyc cyc;
  int smem = 0, at = minlevel - 1;
  cycle_plan(H, level, minlevel, nsmooth, cyc, &smem, &at);
  return bx_vcycle_from(H, level, minlevel, nsmooth, fresh, cyc, smem, at);
}

int bx_finish(Hier& H, int finest, long long nparts, int errortype, bool to_host = true) {
  return after_launch(H, launch_norm_finish(H.s, H.d_partial, (int)nparts, H.nrvars, H.L(finest).count, errortype,
                                            H.d_norm, H.d_nonfinite, to_host ? H.h_norm : nullptr));
}

int bx_resid(Hier& H, int finest, int errortype, bool to_host = true) {
  BoxLev& L = B(H, finest);
  Launch sh = shape(L.n[0], L.n[1], L.n[2]);
  BX_LAUNCH(H, sh, k_bx_resid, H.fpool, L, H.b_oqlo, H.b_ofhi, H.b_oflo, H.d_partial);
  return bx_finish(H, finest, ctas(sh), errortype, to_host);
}

int bx_cycle(Hier& H, int finest, int minlevel, int nsmooth, int errortype, bool to_host = true) {
  int r = bx_vcycle(H, finest, minlevel, nsmooth, true);
  if (r) return r;
  BoxLev& L = B(H, finest);
  if (H.ndims == 3 && L.n[1] % 2 == 0) {  // two rows per thread
    Launch sh = shape(L.n[0], L.n[1] / 2, L.n[2]);
    launch_after(k_bx_track_update<3, 2>, sh.g, sh.b, 0, H.s, H.fpool, L, H.b_oqlo, H.d_partial);
    if ((r = after_launch(H, 1))) return r;
    return bx_finish(H, finest, ctas(sh), errortype, to_host);
  }
  Launch sh = shape(L.n[0], L.n[1], L.n[2]);
  BX_LAUNCH(H, sh, k_bx_track_update, H.fpool, L, H.b_oqlo, H.d_partial);
  return bx_finish(H, finest, ctas(sh), errortype, to_host);
}

// ---------------------------------------------------------------------------
// The solve as one graph launch.  MultigridIterations' loop (afasroutines.f90:
// 81-107) with this path's exit test runs on the device: a WHILE node whose
// body is one cycle (V-cycle, tracked-residual update, norm) and a decision
// kernel, followed by an IF node that evaluates the true residual when the
// decision asks for it.  The host enqueues the loop and reads the control
// block once, instead of waiting for every cycle's norm.

constexpr int kLoopMaxCycles = 64;
struct BoxCtl {
  double tol, r_sync;
  int maxv, it, conv, status, nconfirm, pad;
  double res[kLoopMaxCycles];
};
constexpr int kCtlSlotOffset = 16;  // doubles into the hierarchy's pinned slot
static_assert(sizeof(BoxCtl) <= (128 - kCtlSlotOffset) * sizeof(double) &&
                  sizeof(BoxSolveOut) <= (128 - kCtlSlotOffset) * sizeof(double),
              "pinned slot too small");

// after a cycle: the tracked norm decides whether to confirm on the true
// residual (the host loop's test: below the tolerance, 1e5 below the last
// true residual, or the last cycle)
__global__ void k_bx_decide_cycle(BoxCtl* c, const double* __restrict__ norm, const int* __restrict__ nonfinite,
                                  cudaGraphConditionalHandle hw, cudaGraphConditionalHandle hi) {
  after_previous();
  int it = ++c->it;
  if (c->status || nonfinite[0]) {
    c->status = 1;
    cudaGraphSetConditional(hi, 0);
    cudaGraphSetConditional(hw, 0);
    return;
  }
  double tracked = norm[0];
  bool confirm = tracked < c->tol || tracked < 1e-5 * c->r_sync || it >= c->maxv;
  cudaGraphSetConditional(hi, confirm ? 1u : 0u);
  if (!confirm) c->res[it - 1] = tracked;
}

// after a true residual: converged or the last cycle ends the loop
__global__ void k_bx_decide_true(BoxCtl* c, const double* __restrict__ norm, const int* __restrict__ nonfinite,
                                 cudaGraphConditionalHandle hw) {
  after_previous();
  int it = c->it;
  c->nconfirm++;
  if (nonfinite[0]) {
    c->status = 1;
    cudaGraphSetConditional(hw, 0);
    return;
  }
  double res = norm[0];
  c->r_sync = res;
  c->res[it - 1] = res;
  if (res < c->tol) {
    c->conv = 1;
    cudaGraphSetConditional(hw, 0);
  } else if (it >= c->maxv) {
    cudaGraphSetConditional(hw, 0);
  }
}

// capture what body() enqueues into graph g (a conditional node's body)
int capture_into(Hier& H, cudaGraph_t g, const std::function<int()>& body, long long* nlaunch) {
  cudaError_t e = cudaStreamBeginCaptureToGraph(H.s, g, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal);
  if (e != cudaSuccess) return cuda_fail(e, "cudaStreamBeginCaptureToGraph");
  H.capturing = true;
  H.capture_launches = 0;
  int r = body();
  H.capturing = false;
  *nlaunch = H.capture_launches;
  cudaGraph_t out = nullptr;
  e = cudaStreamEndCapture(H.s, &out);
  if (r) return r;
  if (e != cudaSuccess) return cuda_fail(e, "cudaStreamEndCapture");
  return BSAMG_OK;
}

int box_loop_graph(Hier& H, int finest, int minlevel, int nsmooth, int errortype) {
  auto key = std::make_tuple(finest, minlevel, nsmooth, errortype);
  if (H.box_loop && H.box_loop_key == key) return BSAMG_OK;
  if (H.box_loop) cudaGraphExecDestroy(H.box_loop);
  H.box_loop = nullptr;
  if (!H.box_ctl) {
    cudaError_t e = dev_alloc(H, &H.box_ctl, sizeof(BoxCtl));
    if (e != cudaSuccess) return cuda_fail(e, "device allocation (loop control)");
  }
  BoxCtl* ctl = static_cast<BoxCtl*>(H.box_ctl);
  cudaGraph_t g = nullptr;
  cudaError_t e = cudaGraphCreate(&g, 0);
  if (e != cudaSuccess) return cuda_fail(e, "cudaGraphCreate");
  int r = BSAMG_OK;
  cudaGraphConditionalHandle hw, hi;
  cudaGraphNodeParams wp = {}, ip = {};
  cudaGraphNode_t wn = nullptr;
  do {
    if ((e = cudaGraphConditionalHandleCreate(&hw, g, 1, cudaGraphCondAssignDefault)) != cudaSuccess) break;
    if ((e = cudaGraphConditionalHandleCreate(&hi, g, 0, cudaGraphCondAssignDefault)) != cudaSuccess) break;
    wp.type = cudaGraphNodeTypeConditional;
    wp.conditional.handle = hw;
    wp.conditional.type = cudaGraphCondTypeWhile;
    wp.conditional.size = 1;
    if ((e = cudaGraphAddNode(&wn, g, nullptr, nullptr, 0, &wp)) != cudaSuccess) break;
    cudaGraph_t body = wp.conditional.phGraph_out[0];
    // the cycle, its decision, then the IF node on what was captured
    r = capture_into(H, body, [&]() -> int {
      int rr = bx_cycle(H, finest, minlevel, nsmooth, errortype, false);
      if (rr) return rr;
      launch_after(k_bx_decide_cycle, 1, 1, 0, H.s, ctl, H.d_norm, H.d_nonfinite, hw, hi);
      if ((rr = after_launch(H, 1))) return rr;
      cudaStreamCaptureStatus st;
      cudaGraph_t cg = nullptr;
      const cudaGraphNode_t* deps = nullptr;
      size_t nd = 0;
      cudaError_t ce = cudaStreamGetCaptureInfo(H.s, &st, nullptr, &cg, &deps, nullptr, &nd);
      if (ce != cudaSuccess) return cuda_fail(ce, "cudaStreamGetCaptureInfo");
      ip.type = cudaGraphNodeTypeConditional;
      ip.conditional.handle = hi;
      ip.conditional.type = cudaGraphCondTypeIf;
      ip.conditional.size = 1;
      cudaGraphNode_t in = nullptr;
      ce = cudaGraphAddNode(&in, cg, deps, nullptr, nd, &ip);
      if (ce != cudaSuccess) return cuda_fail(ce, "cudaGraphAddNode(if)");
      ce = cudaStreamUpdateCaptureDependencies(H.s, &in, nullptr, 1, cudaStreamSetCaptureDependencies);
      if (ce != cudaSuccess) return cuda_fail(ce, "cudaStreamUpdateCaptureDependencies");
      return BSAMG_OK;
    }, &H.box_loop_n1);
    if (r) break;
    r = capture_into(H, ip.conditional.phGraph_out[0], [&]() -> int {
      int rr = bx_resid(H, finest, errortype, false);
      if (rr) return rr;
      launch_after(k_bx_decide_true, 1, 1, 0, H.s, ctl, H.d_norm, H.d_nonfinite, hw);
      return after_launch(H, 1);
    }, &H.box_loop_n2);
    if (r) break;
    e = cudaGraphInstantiate(&H.box_loop, g, 0);
  } while (0);
  cudaGraphDestroy(g);
  if (r) return r;
  if (e != cudaSuccess) {
    cudaGetLastError();
    H.box_loop = nullptr;
    return cuda_fail(e, "conditional solve graph");
  }
  H.box_loop_key = key;
  return BSAMG_OK;
}

}  // namespace

bool box_eligible(const Hier& H, bool periodic_single) {
  // the box path's split/merge address q with one ghost layer
  // the box kernels carry CH's equations: only a plugin that declares the
  // box path (CH) takes it
  const Plugin* pl = find_plugin(H.problem);
  if (!pl || !pl->box || !periodic_single || H.mbc != 1) return false;
  for (int l = H.minlevel; l <= H.maxlevel; l++) {
    const HostPatch& P = H.patches[H.L(l).patches[0]];
    for (int d = 0; d < H.ndims; d++) {
      if (P.mx[d] % 2) return false;
      if (l > H.minlevel && P.mx[d] != 2 * H.patches[P.parent].mx[d]) return false;
    }
    // cell indices (both colours) are 32-bit
    if ((long long)P.mx[0] * P.mx[1] * P.mx[2] >= (1LL << 31)) return false;
  }
  return true;
}

// float pool of the box path: per level e, g, pb (not on the finest level,
// where pb is qhi(phi)), ec (below the finest); on the finest level qhi,
// qlo, fhi, flo
void box_coefficients(Hier& H) {
  H.box_plan.reset();  // it holds them
  for (int l = H.maxlevel; l >= H.minlevel; l--) {
    const HostPatch& P = H.patches[H.L(l).patches[0]];
    BoxLev& L = H.blev[l + kMaxDepth];
    double c[4];
    coefficients(H, P.dx[0], c);
    L.c0 = (float)c[0];
    L.c1 = (float)c[1];
    L.tmp3 = (float)c[2];
    L.a12 = (float)c[3];
    L.c0h = (float)c[0];
    L.c0l = (float)(c[0] - (double)L.c0h);
    L.c1h = (float)c[1];
    L.c1l = (float)(c[1] - (double)L.c1h);
    for (int x = 0; x < 4; x++) L.cd[x] = c[x];
  }
}

size_t box_layout(Hier& H) {
  if (cudaDeviceGetAttribute(&H.box_sms, cudaDevAttrMultiProcessorCount, H.ctx->device) != cudaSuccess ||
      H.box_sms <= 0)
    H.box_sms = 1;
  long long o = 0;
  auto al = [](long long x) { return (x + 63) & ~63LL; };
  for (int l = H.maxlevel; l >= H.minlevel; l--) {
    const HostPatch& P = H.patches[H.L(l).patches[0]];
    BoxLev& L = H.blev[l + kMaxDepth];
    for (int d = 0; d < 3; d++) L.n[d] = P.mx[d];
    L.hh = P.mx[0] / 2;
    L.half = (long long)P.mx[0] * P.mx[1] * P.mx[2] / 2;
    L.oe = o; o = al(o + 4 * L.half);
    L.og = o; o = al(o + 4 * L.half);
    if (l == H.maxlevel) {
      L.opb = o; o = al(o + 4 * L.half);    // qhi (both variables)
      H.b_oqlo = o; o = al(o + 4 * L.half);
      H.b_ofhi = o; o = al(o + 2 * L.half);
      H.b_oflo = o; o = al(o + 2 * L.half);
      L.oec = -1;
    } else {
      L.opb = o; o = al(o + 2 * L.half);
      L.oec = o; o = al(o + 4 * L.half);
    }
    L.oe2 = -1;
    if (l > H.minlevel && smooth_fits(H, L)) {  // the one-pass smoothing's output
      L.oe2 = o;
      o = al(o + 4 * L.half);
    }
  }
  box_coefficients(H);
  const BoxLev& F = H.blev[H.maxlevel + kMaxDepth];
  H.b_partials = (size_t)ctas(shape(F.n[0], F.n[1], F.n[2]));
  return (size_t)o;
}

int box_enq_relax(Hier& H, int level, int ipass) { return bx_relax(H, level, ipass - 1, 0); }

int box_smoother_colours(const Hier& H, int level) {
  return level > H.minlevel && smooth_applies(H, H.blev[level + kMaxDepth], 2) ? 4 : 1;
}

int box_enq_smoother(Hier& H, int level, int ipass) {
  if (box_smoother_colours(H, level) == 4) return bx_smooth(H, B(H, level), B(H, level).oe2, false);
  return bx_relax(H, level, ipass - 1, 0);
}

int box_iterations(Hier& H, int finest, int minlevel, int nsmooth, int maxvcycles, double tol, int errortype,
                   int strict, int* ncycles, double* residuals) {
  if (finest != H.maxlevel || minlevel < H.minlevel) return BSAMG_ERR_UNSUPPORTED;
  const HostPatch& P = H.patches[H.L(finest).patches[0]];
  BoxLev& L = B(H, finest);
  Launch sh = shape(L.hh, L.n[1], L.n[2]);
  bool warm = H.box_g_valid;  // g is the residual at this q: update it for the new f
  H.box_g_valid = false;
  if (maxvcycles >= 1 && maxvcycles <= kSolveMaxCycles) {  // one launch where the finest level fits the cluster
    Cyc cyc;
    int smem = 0;
    if (solve_plan(H, finest, minlevel, nsmooth, cyc, &smem)) {
      const BoxSolve bs{H.b_oqlo, H.b_ofhi, H.b_oflo, P.oq, P.oqold, P.sq, P.qn[0], P.qn[1], tol,
                        H.L(finest).count, maxvcycles, errortype, warm ? 1 : 0};
      BoxSolveOut* out = reinterpret_cast<BoxSolveOut*>(H.h_norm + kCtlSlotOffset);
      auto k = H.ndims == 2 ? k_bx_solve<2> : k_bx_solve<3>;
      cudaError_t ce = launch_cluster(k, cyc.ctas, kCycThreads, smem, H.s, H.fpool, H.pool, cyc, L, bs, out);
      if (ce != cudaSuccess) return cuda_fail(ce, "box solve launch");
      int r = after_launch(H, 1);
      if (r || (r = enq_fill_down(H, 2, finest, minlevel))) return r;
      if ((r = stream_wait(H))) return r;
      if (out->status) return BSAMG_ERR_NONFINITE;
      if (residuals)
        for (int n = 0; n < out->it; n++) residuals[n] = out->res[n];
      const bool conv = out->conv != 0;
      if (ncycles) *ncycles = conv ? out->it : maxvcycles;
      H.box_g_valid = true;
      return !conv && strict ? BSAMG_ERR_NOT_CONVERGED : BSAMG_OK;
    }
  }
  // the whole solve as one graph launch when the loop fits its control block
  bool loop = maxvcycles >= 1 && maxvcycles <= kLoopMaxCycles && !H.box_loop_off;
  if (loop) {
    int rl = box_loop_graph(H, finest, minlevel, nsmooth, errortype);
    if (rl == BSAMG_ERR_CUDA && !H.box_loop) {
      H.box_loop_off = true;  // conditional graphs unavailable: the host loop below
      loop = false;
    } else if (rl) {
      return rl;
    }
  }
  int r;
  if (warm) {
    BX_LAUNCH(H, sh, k_bx_split_warm, H.pool, P.oq, P.oqold, P.sq, P.qn[0], P.qn[1], H.fpool, L, H.b_oqlo, H.b_ofhi,
              H.b_oflo, H.d_partial);
    r = bx_finish(H, finest, ctas(sh), errortype, !loop);
  } else {
    BX_LAUNCH(H, sh, k_bx_split, H.pool, P.oq, P.oqold, P.sq, P.qn[0], P.qn[1], H.fpool, L, H.b_oqlo, H.b_ofhi,
              H.b_oflo);
    r = bx_resid(H, finest, errortype, !loop);
  }
  if (r) return r;
  bool conv = false;
  int it = 0;
  if (loop) {
    // control block: the tolerance and cycle limit from the host, the
    // starting residual and its finiteness from the device
    BoxCtl* hc = reinterpret_cast<BoxCtl*>(H.h_norm + kCtlSlotOffset);
    BoxCtl* dc = static_cast<BoxCtl*>(H.box_ctl);
    hc->tol = tol;
    hc->maxv = maxvcycles;
    hc->it = hc->conv = hc->status = hc->nconfirm = 0;
    cudaError_t ce = cudaMemcpyAsync(dc, hc, offsetof(BoxCtl, res), cudaMemcpyHostToDevice, H.s);
    if (ce == cudaSuccess) ce = cudaMemcpyAsync(&dc->r_sync, H.d_norm, sizeof(double), cudaMemcpyDeviceToDevice, H.s);
    if (ce == cudaSuccess) ce = cudaMemcpyAsync(&dc->status, H.d_nonfinite, sizeof(int), cudaMemcpyDeviceToDevice, H.s);
    if (ce == cudaSuccess) ce = cudaGraphLaunch(H.box_loop, H.s);
    if (ce != cudaSuccess) return cuda_fail(ce, "solve graph");
    // leave the state as the FP64 path leaves it (see below), then read
    // the control block once
    BX_LAUNCH(H, sh, k_bx_merge, H.pool, P.oq, P.sq, P.qn[0], P.qn[1], H.fpool, L, H.b_oqlo);
    if ((r = enq_set_ghost(H, finest, 0))) return r;
    if ((r = enq_fill_down(H, 2, finest, minlevel))) return r;
    ce = cudaMemcpyAsync(hc, dc, sizeof(BoxCtl), cudaMemcpyDeviceToHost, H.s);
    if (ce != cudaSuccess) return cuda_fail(ce, "cudaMemcpyAsync(loop control)");
    if (int rw = stream_wait(H)) return rw;
    H.launches += hc->it * H.box_loop_n1 + hc->nconfirm * H.box_loop_n2;
    if (hc->status) return BSAMG_ERR_NONFINITE;
    it = hc->it;
    conv = hc->conv != 0;
    if (residuals)
      for (int n = 0; n < it; n++) residuals[n] = hc->res[n];
    if (ncycles) *ncycles = conv ? it : maxvcycles;
    H.box_g_valid = true;
    if (!conv && strict) return BSAMG_ERR_NOT_CONVERGED;
    return BSAMG_OK;
  }
  if (int rw = stream_wait(H)) return rw;
  if (*H.h_nonfinite) return BSAMG_ERR_NONFINITE;
  double r_sync = H.h_norm[0];
  Hier::GraphRec *gc = nullptr, *gv = nullptr;
  auto key = [&](int m) { return std::make_tuple(m, finest, minlevel, nsmooth, errortype); };
  if ((r = capture_graph(H, key(21), [&] { return bx_cycle(H, finest, minlevel, nsmooth, errortype); }, &gc)))
    return r;
  if ((r = capture_graph(H, key(22), [&] { return bx_resid(H, finest, errortype); }, &gv))) return r;
  for (it = 1; it <= maxvcycles; it++) {
    if ((r = replay(H, gc))) return r;
    if (*H.h_nonfinite) return BSAMG_ERR_NONFINITE;
    double tracked = H.h_norm[0], res = tracked;
    // confirm on the true residual when the tracked one says converged, on
    // the last cycle, and once the tracked value is 1e5 below the residual
    // it started from (where FP32 rounding of g - M(e) stops being negligible)
    if (tracked < tol || tracked < 1e-5 * r_sync || it == maxvcycles) {
      if ((r = replay(H, gv))) return r;
      if (*H.h_nonfinite) return BSAMG_ERR_NONFINITE;
      res = H.h_norm[0];
      r_sync = res;
      if (residuals) residuals[it - 1] = res;
      if (res < tol) {
        conv = true;
        break;
      }
      continue;
    }
    if (residuals) residuals[it - 1] = res;
  }
  if (ncycles) *ncycles = conv ? it : maxvcycles;
  // leave the state as the FP64 path leaves it: q in FP64 with fresh ghosts
  // and the coarse levels restricted from the finest (FillDown,
  // afasroutines.f90:83)
  BX_LAUNCH(H, sh, k_bx_merge, H.pool, P.oq, P.sq, P.qn[0], P.qn[1], H.fpool, L, H.b_oqlo);
  if ((r = enq_set_ghost(H, finest, 0))) return r;
  if ((r = enq_fill_down(H, 2, finest, minlevel))) return r;
  // the loop ends on a true residual (converged, or the last cycle's check)
  H.box_g_valid = true;
  if (!conv && strict) return BSAMG_ERR_NOT_CONVERGED;
  return BSAMG_OK;
}

}  // namespace bsamg
