// Cell addressing and the undivided Laplacian, shared by the kernels of both
// paths and by the plugins' device code.
#pragma once
#include "fp64int.cuh"
#include "internal.h"

namespace bsamg {

// offset of Fortran cell (i,j,k) (lower bound 0) in a ghosted plane of
// extents n
template <int DIM>
__device__ __forceinline__ long long gofs(const int* n, int i, int j, int k) {
  if (DIM == 2) return (long long)j * n[0] + i;
  return ((long long)k * n[1] + j) * n[0] + i;
}
// offset of Fortran cell (i,j,k) (lower bound 1) in an interior plane
template <int DIM>
__device__ __forceinline__ long long iofs(const int* mx, int i, int j, int k) {
  if (DIM == 2) return (long long)(j - 1) * mx[0] + (i - 1);
  return ((long long)(k - 1) * mx[1] + (j - 1)) * mx[0] + (i - 1);
}

// ULap2D / ULap3D, LIBRARY/gridutilities.f90:50-72, :372-399
// In the FP64 part of a plugin (the reference's rounding) the 3D sum runs on
// the integer pipe: the FP64 unit bounds every kernel that evaluates it.
template <int DIM, typename T>
__device__ __forceinline__ T ulap(const T* a, long long c, long long sy, long long sz) {
#ifdef BSAMG_PART_FP64
  if constexpr (DIM == 3 && sizeof(T) == sizeof(double))
    return fxp::lap6({a[c + 1], a[c - 1], a[c + sy], a[c - sy], a[c + sz], a[c - sz]}, a[c]);
#endif
  if (DIM == 2) return a[c + 1] + a[c - 1] + a[c + sy] + a[c - sy] - T(4) * a[c];
  return a[c + 1] + a[c - 1] + a[c + sy] + a[c - sy] + a[c + sz] + a[c - sz] - T(6) * a[c];
}

// The quotients a0/b and a1/b, each bit-identical to the IEEE
// round-to-nearest division: on the integer pipe for 1 <= b < 2^400 and
// 2^-400 <= |a| < 2^400, and `/` for everything else (zeros, tiny or huge
// values, NaN and Inf); checked on the GPU over random and edge-case operands.
__device__ __forceinline__ void div2_rn(double a0, double a1, double b, double& q0, double& q1) {
  fxp::quot2(a0, a1, b, q0, q1);
}

__device__ __forceinline__ double cube(double c) { return c * c * c; }  // CH/problem.f90:918
__device__ __forceinline__ double sqr(double c) { return c * c; }       // CH/problem.f90:931

// map a unit of a colour work list to an interior cell; false if the slot is
// past the end of its row (odd mx) or past the patch.  The colour test is the
// reference loop start i = 1 + MODULO(j(+k)+ipass, 2) (CH/problem.f90:350,
// :591).
template <int DIM>
__device__ __forceinline__ bool color_cell(const PatchDev& p, int t, int ipass, int& i, int& j, int& k) {
  int hx = (p.mx[0] + 1) >> 1;
  int row = t / hx;
  int s = t - row * hx;
  if (DIM == 2) {
    j = row + 1;
    k = 1;
    if (j > p.mx[1]) return false;
    i = 1 + ((j + ipass) & 1) + 2 * s;
  } else {
    j = row % p.mx[1] + 1;
    k = row / p.mx[1] + 1;
    if (k > p.mx[2]) return false;
    i = 1 + ((k + j + ipass) & 1) + 2 * s;
  }
  return i <= p.mx[0];
}

template <int DIM>
__device__ __forceinline__ bool interior_cell(const int* mx, int t, int& i, int& j, int& k) {
  i = t % mx[0] + 1;
  int r = t / mx[0];
  if (DIM == 2) {
    j = r + 1;
    k = 1;
    return j <= mx[1];
  }
  j = r % mx[1] + 1;
  k = r / mx[1] + 1;
  return k <= mx[2];
}

// cell t of a ghosted array of extents n whose indices start at -gs
template <int DIM>
__device__ __forceinline__ bool ghosted_cell(const int* n, int gs, int t, int& i, int& j, int& k) {
  i = t % n[0] - gs;
  int r = t / n[0];
  if (DIM == 2) {
    j = r - gs;
    k = 0;
    return r < n[1];
  }
  j = r % n[1] - gs;
  k = r / n[1];
  bool ok = k < n[2];
  k -= gs;
  return ok;
}

// The sums of a warp's NV FP64 values a lane -> red[v][w], each the tree of
// shfl_down(16, 8, 4, 2, 1) bit for bit.  An FP64 add takes the unit 64
// cycles for however many lanes: two to four variables share the adds, each
// half (quarter) of the warp holding one of them after the first steps (5
// adds for 2 variables instead of 10, 6 for 3 instead of 15).  A warp whose
// lanes all hold zero adds nothing.
template <int NV, int W>
__device__ __forceinline__ void warp_sums(const double (&s)[NV], double (*red)[W], int w, int lane, bool any) {
  if (!any) {
    if (lane < NV) red[lane][w] = 0.0;
    return;
  }
  auto peer = [](double x, int o) { return __shfl_xor_sync(0xffffffffu, x, o); };
  if constexpr (NV < 2 || NV > 4) {
    for (int v = 0; v < NV; v++) {
      double t = s[v];
      for (int o = 16; o > 0; o >>= 1) t = __dadd_rn(t, peer(t, o));
      if (lane == 0) red[v][w] = t;
    }
  } else {
    const bool h = lane & 16, q = lane & 8;
    double r = __dadd_rn(h ? s[1] : s[0], peer(h ? s[0] : s[1], 16));  // variable 0 | 1
    if constexpr (NV == 2) {
      r = __dadd_rn(r, peer(r, 8));
    } else {
      double r2;  // variable 2 (| 3)
      if constexpr (NV == 4) r2 = __dadd_rn(h ? s[3] : s[2], peer(h ? s[2] : s[3], 16));
      else r2 = __dadd_rn(s[2], peer(s[2], 16));
      const double send = q ? r : r2;
      r = __dadd_rn(q ? r2 : r, peer(send, 8));
    }
    for (int o = 4; o > 0; o >>= 1) r = __dadd_rn(r, peer(r, o));
    const int v = (h ? 1 : 0) + (NV > 2 && q ? 2 : 0);
    if ((lane & 7) == 0 && (NV > 2 || !q) && v < NV && !(NV == 3 && h && q)) red[v][w] = r;
  }
}

}  // namespace bsamg
