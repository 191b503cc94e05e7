// Uniform levels: the levels <= 0 of every hierarchy are one patch that
// covers the domain (RootInit/InitSeed, LIBRARY/bsamroutines.f90:226-510), so
// SetGhost on them (boundary.f90:67-97) is a pure copy: every ghost cell is
// one interior cell's value, shifted by qpo across the periodic x faces and
// passed through the plugin's UserBC once per physical face it lies beyond.
// The operations here push those images when they write the interior cell,
// so a level needs no ghost pass of its own: a colour sweep reads the ghosts
// the previous one left (before the first: k_uni_walls), and the images it
// writes are of its own colour, which no cell of that colour reads (periodic
// extents are even; a physical face's ghost is read only by the cell it
// images).  Every cell computes what
// the stand-alone kernel of the operation computes, in the same order.
//
// The same operations run in two forms: as one launch per operation over a
// level in global memory, and as the whole V-cycle of the coarse levels in
// one launch of a thread-block cluster, each CTA holding a slab of rows (the
// slowest dimension) of every level in its shared memory with one halo row
// at each side.  There the halo rows are pushed too, into the neighbour's
// shared memory, so all reads are local and a phase costs one cluster
// barrier; levels too small to share out are held by CTA 0 alone.
//
// Included by the FP64 part (T = double, --fmad=false: the reference's
// rounding) and by the mixed part (T = float: the correction cycle) of every
// plugin; TR is the trait of one of the two (Uni64, Uni32).
#pragma once
#include <cuda_runtime.h>

#include "cellops.cuh"
#include "launch.h"
#include "plugin.h"

namespace bsamg {
namespace uni {

extern __shared__ __align__(16) unsigned char uni_smem[];

// a / d and a % d for 0 <= a < 2^31: the high half of a * ceil(2^32 / d) is
// the quotient or one above it
__device__ __forceinline__ void fdivmod(int a, const UniDiv& d, int& q, int& r) {
  q = d.m ? (int)__umulhi((unsigned)a, d.m) : a;
  r = a - q * d.d;
  if (r < 0) {
    q--;
    r += d.d;
  }
}

// A ghosted array of a level (or of its coarse image) as one CTA holds it:
// interior extents, rows r0+1 .. r0+nr (global, 1-based, of the slowest
// dimension) of N in local rows 1 .. nr, and the strides of the next x row,
// the next plane (3D) and the next variable.
struct Geo {
  int n0, n1, N, r0, nr;
  int sy, sz, sq;
};

// How the rows of a level are dealt to the CTAs, as one of them sees it:
// whether the level is shared out, whether it holds the domain's first and
// last row, and the ranks below and above (around the domain) with the rows
// of the one below.
struct Part {
  bool shared, first, last;
  int lo, hi, lo_rows;
};

// One level as one CTA (or one launch) sees it: q, f, the coarse image c of
// q, and x, the frozen data beside it (qold in q's layout, or base planes in
// f's).  Pointers are to cell (0,0,0) of variable 1.
template <typename T>
struct View {
  T *q, *f, *c, *x;
  Geo g, gc;
  int sf;
  const UniDim* d;
};

template <typename T>
__device__ __forceinline__ T* on_rank(T* p, int rank) {
  return static_cast<T*>(__cluster_map_shared_rank(static_cast<void*>(p), rank));
}

template <int DIM>
__device__ __forceinline__ int gcell(const Geo& g, int i, int j, int k) {
  return DIM == 2 ? j * g.sy + i : k * g.sz + j * g.sy + i;
}
template <int DIM>
__device__ __forceinline__ int icell(const Geo& g, int i, int j, int k) {
  return DIM == 2 ? (j - 1) * g.n0 + (i - 1) : ((k - 1) * g.n1 + (j - 1)) * g.n0 + (i - 1);
}

// Cell t of one colour (ipass) of the level's rows; false past a row's end
template <int DIM>
__device__ __forceinline__ bool colour_unit(const Geo& g, const UniDim& d, int t, int colour, int& i, int& j, int& k) {
  int r, s, par;
  fdivmod(t, d.hx, r, s);
  if (DIM == 3) {
    fdivmod(r, d.n1, k, j);
    j++;
    k++;
    par = j + k + g.r0;
  } else {
    j = r + 1;
    k = 1;
    par = j + g.r0;
  }
  i = 1 + ((par + colour) & 1) + 2 * s;
  return i <= g.n0;
}
template <int DIM>
__device__ __forceinline__ int colour_units(const Geo& g) {
  return ((g.n0 + 1) >> 1) * (DIM == 3 ? g.n1 : 1) * g.nr;
}
// interior cell t of extents n0 x (n1 x) rows
template <int DIM>
__device__ __forceinline__ void inner_unit(const UniDiv& n0, const UniDiv& n1, int t, int& i, int& j, int& k) {
  int r;
  fdivmod(t, n0, r, i);
  i++;
  k = 1;
  if (DIM == 3) {
    fdivmod(r, n1, k, j);
    j++;
    k++;
  } else {
    j = r + 1;
  }
}
template <int DIM>
__device__ __forceinline__ int inner_units(const Geo& g) {
  return g.n0 * (DIM == 3 ? g.n1 : 1) * g.nr;
}

// Write the images of interior cell (i, j, k) of a whole level, whose NV
// values are w: one ghost per face it touches and, with `full`, the edge and
// corner ghosts too (stencils read only the face ghosts; the prolongation
// reads the rest).  Every extent is at least 2, so a cell has at most one
// image per dimension and the images are the nonempty subsets of those.
template <class TR, int DIM>
__device__ __forceinline__ void push(typename TR::T* base, const Geo& g, int i, int j, int k, const typename TR::T* w,
                                     bool full, const UniBC& bc, const typename TR::Par& par) {
  using T = typename TR::T;
  const int x[3] = {i, j, DIM == 3 ? k : 1};
  const int n[3] = {g.n0, DIM == 3 ? g.n1 : g.N, DIM == 3 ? g.N : 2};
  const int st[3] = {1, g.sy, g.sz};
  int flags = 0, delta[3];
#pragma unroll
  for (int d = 0; d < DIM; d++) {
    const bool lo = x[d] == 1, hi = x[d] == n[d];
    if (lo || hi) flags |= 1 << d;
    const int to = bc.phys[d] ? (lo ? 0 : n[d] + 1) : (lo ? n[d] + 1 : 0);
    delta[d] = (to - x[d]) * st[d];
  }
  if (!flags) return;
  const int at = gcell<DIM>(g, i, j, k);
#pragma unroll
  for (int m = 1; m < (1 << DIM); m++) {
    if ((m & flags) != m || (!full && (m & (m - 1)))) continue;
    int b = at, nb = 0;
#pragma unroll
    for (int d = 0; d < DIM; d++)
      if (m & (1 << d)) {
        b += delta[d];
        nb += bc.phys[d];
      }
    const int sh = (m & 1) && !bc.phys[0] ? (i == 1 ? 1 : 2) : 0;
#pragma unroll
    for (int v = 0; v < TR::NV; v++) {
      T u = TR::shift(w[v], sh, v, par);
#pragma unroll
      for (int z = 0; z < DIM; z++)
        if (z < nb) u = TR::wall(u, bc.mask, v);
      base[v * g.sq + b] = u;
    }
  }
}

// One colour of a whole level's relaxation; the images of its cells follow
template <class TR, int DIM>
__device__ __forceinline__ void relax(const View<typename TR::T>& V, int ipass, bool full, int t0, int nt,
                                      const PatchDev& P, const UniBC& bc, const typename TR::Par& par) {
  const Geo& g = V.g;
  const int units = colour_units<DIM>(g);
  for (int t = t0; t < units; t += nt) {
    int i, j, k;
    if (!colour_unit<DIM>(g, *V.d, t, ipass & 3, i, j, k)) continue;
    const int c = gcell<DIM>(g, i, j, k);
    TR::template relax<DIM>(V, c, icell<DIM>(g, i, j, k), ipass, P, par);
    typename TR::T w[TR::NV];
#pragma unroll
    for (int v = 0; v < TR::NV; v++) w[v] = V.q[v * g.sq + c];
    push<TR, DIM>(V.q, g, i, j, k, w, full, bc, par);
  }
}

// x 2^K and, in 3D, 3 x: FP64 on the integer pipe (fp64int.cuh; a chain of
// FP64 instructions bounds the small levels, their number the large ones)
template <int K>
__device__ __forceinline__ double scaled(double x) {
  return fxp::scaled<K>(x);
}
template <int K>
__device__ __forceinline__ float scaled(float x) {
  return x * (K < 0 ? 1.0f / (1 << (K < 0 ? -K : 0)) : 1.0f * (1 << (K > 0 ? K : 0)));
}
template <int DIM>
__device__ __forceinline__ double triple(double x) {
  if constexpr (DIM == 3) return fxp::triple(x);
  return 3.0 * x;
}
template <int DIM>
__device__ __forceinline__ float triple(float x) {
  return 3.0f * x;
}

// mean of the 4 (8) fine values whose highest cell is a[0], summed in the
// order of Restriction2D/3D (gridutilities.f90:103-126, :437-466)
template <int DIM, typename T>
__device__ __forceinline__ T mean(const T* a, int sy, int sz) {
  T s = a[0] + a[-1] + a[-sy] + a[-sy - 1];
  if (DIM == 3) s = s + a[-sz] + a[-sz - 1] + a[-sz - sy] + a[-sz - sy - 1];
  return scaled<DIM == 2 ? -2 : -3>(s);
}

// RestrictSolution (afasroutines.f90:610-652): the coarse image and the
// parent's q take R(q), with SetGhost of the parent (face images) and
// GetCoarseGhostPoints (boundary.f90:957-1015) of the image
template <class TR, int DIM>
__device__ __forceinline__ void restrict_q(const View<typename TR::T>& V, const View<typename TR::T>& U,
                                           int t0, int nt, const UniBC& bc, const typename TR::Par& par) {
  using T = typename TR::T;
  const Geo &g = V.g, &gc = V.gc;
  const int units = inner_units<DIM>(gc);
  for (int t = t0; t < units; t += nt) {
    int ci, cj, ck;
    inner_unit<DIM>(V.d->c0, V.d->c1, t, ci, cj, ck);
    const int f = gcell<DIM>(g, 2 * ci, 2 * cj, 2 * ck);
    T w[TR::NV];
#pragma unroll
    for (int v = 0; v < TR::NV; v++) {
      w[v] = mean<DIM>(V.q + v * g.sq + f, g.sy, g.sz);
      V.c[v * gc.sq + gcell<DIM>(gc, ci, cj, ck)] = w[v];
      U.q[v * U.g.sq + gcell<DIM>(U.g, ci, cj, ck)] = w[v];
    }
    push<TR, DIM>(V.c, gc, ci, cj, ck, w, true, bc, par);
    push<TR, DIM>(U.q, U.g, ci, cj, ck, w, false, bc, par);
  }
}

// CoarseLoadingFunction with Residual (afasroutines.f90:673-736, :817-857) of
// a whole level: parent f = R(f - Op(q)) + Op_2h(coarse image); rf (FP64) is
// stored in the level's own interior layout.
template <class TR, int DIM>
__device__ __forceinline__ void coarse_load(const View<typename TR::T>& V, const View<typename TR::T>& U,
                                            typename TR::T* rf, int t0, int nt, const PatchDev& P, const PatchDev& PU,
                                            const typename TR::Par& par) {
  using T = typename TR::T;
  const Geo &g = V.g, &gc = V.gc;
  const int units = inner_units<DIM>(gc);
  for (int t = t0; t < units; t += nt) {
    int ci, cj, ck;
    inner_unit<DIM>(V.d->c0, V.d->c1, t, ci, cj, ck);
    T R[TR::NV];
    // the integer Laplacians of eight cells in a row do not fit the instruction
    // cache, nor twice the CTAs the registers (256^3 FP64 step: unrolled 53.1
    // ms, rolled 50.4)
    constexpr int kUnroll = DIM == 3 && sizeof(T) == 8 ? 1 : 1 << DIM;
#pragma unroll(kUnroll)
    for (int m = 0; m < (1 << DIM); m++) {
      const int i = 2 * ci - (m & 1), j = 2 * cj - ((m >> 1) & 1), k = DIM == 3 ? 2 * ck - (m >> 2) : 1;
      const int c = gcell<DIM>(g, i, j, k), fc = icell<DIM>(g, i, j, k);
      T r[TR::NV];
      TR::template op<DIM>(V.q, c, g, V, c, fc, P, par, r);
#pragma unroll
      for (int v = 0; v < TR::NV; v++) {
        const T e = V.f[v * V.sf + fc] - r[v];
        if (TR::kStoreRf) rf[v * V.sf + fc] = e;
        R[v] = m ? R[v] + e : e;
      }
    }
    T cr[TR::NV];
    const int fu = icell<DIM>(U.g, ci, cj, ck);
    TR::template op<DIM>(V.c, gcell<DIM>(gc, ci, cj, ck), gc, U, gcell<DIM>(U.g, ci, cj, ck), fu, PU, par, cr);
#pragma unroll
    for (int v = 0; v < TR::NV; v++) U.f[v * U.sf + fu] = scaled<DIM == 2 ? -2 : -3>(R[v]) + cr[v];
  }
}

// The value of the parent's ghosted cell (i, j, k) of variable v, its edge
// and corner ghosts from their interior cell (they are refreshed only where
// something reads them)
template <class TR, int DIM>
__device__ __forceinline__ typename TR::T ghosted_value(const typename TR::T* q, const Geo& g, int i, int j, int k,
                                                        int v, const UniBC& bc, const typename TR::Par& par) {
  int nb = 0, sh = 0;
  auto src = [&](int x, int n, int d) {
    if (x >= 1 && x <= n) return x;
    if (bc.phys[d]) {
      nb++;
      return x < 1 ? 1 : n;
    }
    if (d == 0) sh = x < 1 ? 2 : 1;
    return x < 1 ? n : 1;
  };
  const int si = src(i, g.n0, 0), sj = src(j, DIM == 3 ? g.n1 : g.N, 1), sk = DIM == 3 ? src(k, g.N, 2) : 1;
  typename TR::T u = TR::shift(q[v * g.sq + gcell<DIM>(g, si, sj, sk)], sh, v, par);
#pragma unroll
  for (int z = 0; z < DIM; z++)
    if (z < nb) u = TR::wall(u, bc.mask, v);
  return u;
}

template <class TR, int DIM>
__device__ __forceinline__ typename TR::T slab_value(const typename TR::T* q, const Geo& g, const Part& pt, int i,
                                                     int j, int k, int v, const UniBC& bc,
                                                     const typename TR::Par& par);

// CorrectFine step 1 (afasroutines.f90:892-895, :934-938): the coarse image
// becomes parent q - image, ghosts (and a slab's halo rows) included.  WHOLE:
// a whole level, whose parent's edge and corner ghosts may be stale; else pu
// is the parent's part.
template <class TR, int DIM, bool WHOLE>
__device__ __forceinline__ void correct_a(const View<typename TR::T>& V, const View<typename TR::T>& U,
                                          const Part& pu, int t0, int nt, const UniBC& bc,
                                          const typename TR::Par& par) {
  const Geo& gc = V.gc;
  const int units = (gc.n0 + 2) * (DIM == 3 ? gc.n1 + 2 : 1) * (gc.nr + 2);
  const int up = gc.r0 - U.g.r0;
  for (int t = t0; t < units; t += nt) {
    int r, i, j, k = 0;
    fdivmod(t, V.d->ce0, r, i);
    if (DIM == 3) fdivmod(r, V.d->ce1, k, j);
    else j = r;
    const int c = gcell<DIM>(gc, i, j, k);
    const int pj = DIM == 2 ? j + up : j, pk = k + up;
#pragma unroll
    for (int v = 0; v < TR::NV; v++) {
      const typename TR::T u = WHOLE ? ghosted_value<TR, DIM>(U.q, U.g, i, pj, pk, v, bc, par)
                                     : slab_value<TR, DIM>(U.q, U.g, pu, i, pj, pk, v, bc, par);
      V.c[v * gc.sq + c] = u - V.c[v * gc.sq + c];
    }
  }
}

// CorrectFine step 2 and SetGhost's face images: q += Bi/TriLinProlongationP1
// (coarse image) (gridutilities.f90:156-195, :510-566) on the interior of a
// whole level.  One thread per coarse index 0 .. cmx in every dimension (see
// u_correct_b).  INLINE_A: the image still holds R(q) and step 1 is done on
// the fly (the correction cycle, whose coarse image nothing else reads).
template <class TR, int DIM, bool INLINE_A>
__device__ __forceinline__ void correct_b(const View<typename TR::T>& V, const View<typename TR::T>& U, int t0, int nt,
                                          const UniBC& bc, const typename TR::Par& par) {
  using T = typename TR::T;
  const Geo &g = V.g, &gc = V.gc;
  const int units = (gc.n0 + 1) * (DIM == 3 ? gc.n1 + 1 : 1) * (gc.nr + 1);
  constexpr int NZ = DIM == 3 ? 2 : 1;
  for (int t = t0; t < units; t += nt) {
    int r, ci, cj, ck = 0;
    fdivmod(t, V.d->cp0, r, ci);
    if (DIM == 3) fdivmod(r, V.d->cp1, ck, cj);
    else cj = r;
    T out[4 * NZ][TR::NV];
#pragma unroll
    for (int v = 0; v < TR::NV; v++) {
      const T* a = V.c + v * gc.sq;
      auto at = [&](int i, int j, int k) -> T {
        const T x = a[gcell<DIM>(gc, i, j, k)];
        return INLINE_A ? ghosted_value<TR, DIM>(U.q, U.g, i, j, k, v, bc, par) - x : x;
      };
      T b[NZ][2][2];
#pragma unroll
      for (int dz = 0; dz < NZ; dz++)
#pragma unroll
        for (int dy = 0; dy < 2; dy++) {
          const T lo = at(ci, cj + dy, ck + dz), hi = at(ci + 1, cj + dy, ck + dz);
          b[dz][dy][0] = triple<DIM>(lo) + hi;
          b[dz][dy][1] = lo + triple<DIM>(hi);
        }
#pragma unroll
      for (int fy = 0; fy < 2; fy++)
#pragma unroll
        for (int fx = 0; fx < 2; fx++) {
          const T c0 = fy == 0 ? triple<DIM>(b[0][0][fx]) + b[0][1][fx] : b[0][0][fx] + triple<DIM>(b[0][1][fx]);
          if (DIM == 2) {
            out[fy * 2 + fx][v] = scaled<-4>(c0);
          } else {
            const T c1 = fy == 0 ? triple<DIM>(b[NZ - 1][0][fx]) + b[NZ - 1][1][fx]
                                 : b[NZ - 1][0][fx] + triple<DIM>(b[NZ - 1][1][fx]);
            out[fy * 2 + fx][v] = scaled<-6>(triple<DIM>(c0) + c1);
            out[(NZ - 1) * 4 + fy * 2 + fx][v] = scaled<-6>(c0 + triple<DIM>(c1));
          }
        }
    }
    // every fine value is loaded before the first store, which the next load
    // would have to wait for (V.q is both)
    int at[4 * NZ];
#pragma unroll
    for (int m = 0; m < 4 * NZ; m++) {
      const int i = 2 * ci + (m & 1), j = 2 * cj + ((m >> 1) & 1), k = DIM == 3 ? 2 * ck + (m >> 2) : 1;
      const bool in = i >= 1 && i <= g.n0 && j >= 1 && j <= (DIM == 3 ? g.n1 : g.N) && (DIM != 3 || (k >= 1 && k <= g.N));
      at[m] = in ? gcell<DIM>(g, i, j, k) : -1;
#pragma unroll
      for (int v = 0; v < TR::NV; v++)
        if (in) out[m][v] = V.q[v * g.sq + at[m]] + out[m][v];
    }
#pragma unroll
    for (int m = 0; m < 4 * NZ; m++) {
      if (at[m] < 0) continue;
#pragma unroll
      for (int v = 0; v < TR::NV; v++) V.q[v * g.sq + at[m]] = out[m][v];
      push<TR, DIM>(V.q, g, 2 * ci + (m & 1), 2 * cj + ((m >> 1) & 1), DIM == 3 ? 2 * ck + (m >> 2) : 1, out[m], false, bc,
                    par);
    }
  }
}

// FillDownLevel (afasroutines.f90:257-327): fields bit 0: parent q = R(q),
// interior and, with SetGhost, ghosts; bit 1: parent f = R(f)
template <class TR, int DIM>
__device__ __forceinline__ void fill_down(const View<typename TR::T>& V, const View<typename TR::T>& U, int fields,
                                          int t0, int nt, const UniBC& bc, const typename TR::Par& par) {
  using T = typename TR::T;
  const Geo &g = V.g, &gc = V.gc;
  const int units = inner_units<DIM>(gc);
  for (int t = t0; t < units; t += nt) {
    int ci, cj, ck;
    inner_unit<DIM>(V.d->c0, V.d->c1, t, ci, cj, ck);
    if (fields & 1) {
      T w[TR::NV];
#pragma unroll
      for (int v = 0; v < TR::NV; v++) {
        w[v] = mean<DIM>(V.q + v * g.sq + gcell<DIM>(g, 2 * ci, 2 * cj, 2 * ck), g.sy, g.sz);
        U.q[v * U.g.sq + gcell<DIM>(U.g, ci, cj, ck)] = w[v];
      }
      push<TR, DIM>(U.q, U.g, ci, cj, ck, w, true, bc, par);
    }
    if (fields & 2) {
#pragma unroll
      for (int v = 0; v < TR::NV; v++)
        U.f[v * U.sf + icell<DIM>(U.g, ci, cj, ck)] =
            mean<DIM>(V.f + v * V.sf + icell<DIM>(g, 2 * ci, 2 * cj, 2 * ck), g.n0, g.n0 * g.n1);
    }
  }
}

// ghost cell t of the shell of a level: 2D: rows 0 and N+1 whole, then cells
// 0 and n0+1 of the others; 3D: planes 0 and N+1 whole, then the frame of
// the others
template <int DIM>
__device__ __forceinline__ int shell_units(const Geo& g) {
  const int e0 = g.n0 + 2;
  return DIM == 3 ? 2 * e0 * (g.n1 + 2) + g.N * (2 * e0 + 2 * g.n1) : 2 * e0 + 2 * g.N;
}
// WALLS: the ghosts beyond one wall of the cells of colour 2 only (k_uni_walls)
template <class TR, int DIM, bool WALLS = false>
__device__ __forceinline__ void set_ghost(typename TR::T* q, const Geo& g, const UniDim& d, int t0, int nt,
                                          const UniBC& bc, const typename TR::Par& par) {
  const int e0 = g.n0 + 2, cap = DIM == 3 ? e0 * (g.n1 + 2) : e0;
  const int units = shell_units<DIM>(g);
  for (int t = t0; t < units; t += nt) {
    int i, j = 0, row;
    if (t < 2 * cap) {
      const int hi = t >= cap, u = t - hi * cap;
      row = hi ? g.N + 1 : 0;
      if (DIM == 3) fdivmod(u, d.e0, j, i);
      else i = u;
    } else {
      int u;
      if (DIM == 2) {
        u = t - 2 * cap;
        row = (u >> 1) + 1;
        i = (u & 1) ? g.n0 + 1 : 0;
      } else {
        fdivmod(t - 2 * cap, d.ring, row, u);
        row++;
        if (u < 2 * e0) {
          j = u < e0 ? 0 : g.n1 + 1;
          i = u < e0 ? u : u - e0;
        } else {
          j = ((u - 2 * e0) >> 1) + 1;
          i = (u & 1) ? g.n0 + 1 : 0;
        }
      }
    }
    const int jj = DIM == 2 ? row : j, kk = row;
    if (WALLS) {
      const int x[3] = {i, jj, kk}, n[3] = {g.n0, DIM == 3 ? g.n1 : g.N, g.N};
      int beyond = 0, walls = 0, sum = 0;
#pragma unroll
      for (int b = 0; b < DIM; b++) {
        const bool out = x[b] < 1 || x[b] > n[b];
        beyond += out;
        walls += out && bc.phys[b];
        sum += x[b] < 1 ? 1 : (x[b] > n[b] ? n[b] : x[b]);
      }
      if (beyond != 1 || walls != 1 || !(sum & 1)) continue;
    }
#pragma unroll
    for (int v = 0; v < TR::NV; v++)
      q[v * g.sq + gcell<DIM>(g, i, jj, kk)] = ghosted_value<TR, DIM>(q, g, i, jj, kk, v, bc, par);
  }
}

// the view of a whole level in global memory
template <class TR, int DIM>
__device__ __forceinline__ View<typename TR::T> global_view(const PatchDev& p, const UniDim& d,
                                                            const typename TR::Mem& m) {
  View<typename TR::T> V;
  V.g = Geo{p.mx[0], p.mx[1], DIM == 2 ? p.mx[1] : p.mx[2], 0, DIM == 2 ? p.mx[1] : p.mx[2],
            p.qn[0], p.qn[0] * p.qn[1], (int)p.sq};
  V.gc = Geo{p.cmx[0], p.cmx[1], DIM == 2 ? p.cmx[1] : p.cmx[2], 0, DIM == 2 ? p.cmx[1] : p.cmx[2],
             p.cn[0], p.cn[0] * p.cn[1], (int)p.sc};
  V.sf = (int)p.sf;
  V.d = &d;
  TR::bind(V, p, m);
  return V;
}

// ---- one launch per operation over a level in global memory ----

// The patch of a level and its parent's arrive by value (their geometry
// costs no load); the coefficients are read through the table P, so that
// captured graphs survive bsamg_set_params.
#define UNI_T0 (int)(blockIdx.x * kBlock + threadIdx.x), (int)(gridDim.x * kBlock)
template <class TR, int DIM>
__global__ void __launch_bounds__(kBlock) k_uni_relax(const PatchDev* __restrict__ P, typename TR::Mem m, int patch,
                                                      const __grid_constant__ UniPatch p, int ipass, int full, UniBC bc,
                                                      typename TR::Par par) {
  after_previous();
  relax<TR, DIM>(global_view<TR, DIM>(p.p, p.d, m), ipass, full, UNI_T0, P[patch], bc, par);
}
template <class TR, int DIM>
__global__ void __launch_bounds__(kBlock) k_uni_restrict(typename TR::Mem m, const __grid_constant__ UniPatch p,
                                                         const __grid_constant__ UniPatch u, UniBC bc,
                                                         typename TR::Par par) {
  after_previous();
  restrict_q<TR, DIM>(global_view<TR, DIM>(p.p, p.d, m), global_view<TR, DIM>(u.p, u.d, m), UNI_T0, bc, par);
}
template <class TR, int DIM>
__global__ void __launch_bounds__(kBlock) k_uni_load(const PatchDev* __restrict__ P, typename TR::Mem m, int patch,
                                                     const __grid_constant__ UniPatch p, int parent,
                                                     const __grid_constant__ UniPatch u, typename TR::Par par) {
  after_previous();
  coarse_load<TR, DIM>(global_view<TR, DIM>(p.p, p.d, m), global_view<TR, DIM>(u.p, u.d, m), TR::rf(p.p, m), UNI_T0,
                       P[patch], P[parent], par);
}
template <class TR, int DIM>
__global__ void __launch_bounds__(kBlock) k_uni_correct_a(typename TR::Mem m, const __grid_constant__ UniPatch p,
                                                          const __grid_constant__ UniPatch u, UniBC bc,
                                                          typename TR::Par par) {
  after_previous();
  correct_a<TR, DIM, true>(global_view<TR, DIM>(p.p, p.d, m), global_view<TR, DIM>(u.p, u.d, m), Part{}, UNI_T0, bc,
                           par);
}
template <class TR, int DIM>
__global__ void __launch_bounds__(kBlock) k_uni_correct_b(typename TR::Mem m, const __grid_constant__ UniPatch p,
                                                          const __grid_constant__ UniPatch u, UniBC bc,
                                                          typename TR::Par par) {
  after_previous();
  correct_b<TR, DIM, !TR::kStoreRf>(global_view<TR, DIM>(p.p, p.d, m), global_view<TR, DIM>(u.p, u.d, m), UNI_T0, bc,
                                    par);
}
template <class TR, int DIM>
__global__ void __launch_bounds__(kBlock) k_uni_ghost(typename TR::Mem m, const __grid_constant__ UniPatch p, UniBC bc,
                                                      typename TR::Par par) {
  after_previous();
  const View<typename TR::T> V = global_view<TR, DIM>(p.p, p.d, m);
  set_ghost<TR, DIM>(V.q, V.g, p.d, UNI_T0, bc, par);
}
// The ghosts beyond the walls of a level whose ghosts the caller may not have
// set, before its first smoothing.  SetGhost after the first colour's sweep
// refreshes them for the second colour; the sweep here pushes its own
// colour's only.  (The second colour's periodic images are read by the first
// colour alone, which takes them as they are, here and there.)
template <class TR, int DIM>
__global__ void __launch_bounds__(kBlock) k_uni_walls(typename TR::Mem m, const __grid_constant__ UniPatch p, UniBC bc,
                                                      typename TR::Par par) {
  after_previous();
  const View<typename TR::T> V = global_view<TR, DIM>(p.p, p.d, m);
  set_ghost<TR, DIM, true>(V.q, V.g, p.d, UNI_T0, bc, par);
}
template <class TR, int DIM>
__global__ void __launch_bounds__(kBlock) k_uni_fill(typename TR::Mem m, const __grid_constant__ UniPatch p,
                                                     const __grid_constant__ UniPatch u, int fields, UniBC bc,
                                                     typename TR::Par par) {
  after_previous();
  fill_down<TR, DIM>(global_view<TR, DIM>(p.p, p.d, m), global_view<TR, DIM>(u.p, u.d, m), fields, UNI_T0, bc, par);
}

// the table entries of the levels of A in shared memory: a global load
// after a cluster barrier is an L2 round trip, since the barrier's acquire
// discards what L1 holds
__device__ __forceinline__ void stage_table(PatchDev* sp, const PatchDev* __restrict__ P, const UniCycle& A) {
  constexpr int W = (int)(sizeof(PatchDev) / 4);
  for (int q = threadIdx.x; q < A.nl * W; q += blockDim.x) {
    const int x = q / W;
    reinterpret_cast<int*>(&sp[x])[q - x * W] = reinterpret_cast<const int*>(&P[A.L[x].patch])[q - x * W];
  }
  __syncthreads();
}

// FillDown through the levels of A in one CTA (levels too small to fill the GPU)
template <class TR, int DIM>
__global__ void __launch_bounds__(kUniFillThreads) k_uni_fill_small(const PatchDev* __restrict__ P, typename TR::Mem m,
                                                                    const __grid_constant__ UniCycle A, int fields,
                                                                    typename TR::Par par) {
  after_previous();
  __shared__ __align__(16) PatchDev sp[kNLev];
  stage_table(sp, P, A);
  for (int x = 0; x + 1 < A.nl; x++) {
    fill_down<TR, DIM>(global_view<TR, DIM>(sp[x], A.L[x].d, m), global_view<TR, DIM>(sp[x + 1], A.L[x + 1].d, m),
                       fields, threadIdx.x, blockDim.x, A.bc, par);
    __syncthreads();
  }
}

// ---- the V-cycle of the coarse levels in one launch of one cluster ----

__device__ __forceinline__ int my_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return (int)r;
}
__device__ __forceinline__ void cluster_sync() {
  __syncwarp();  // the aligned forms want the warp converged
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Where the images of a slab's first and last row go: a halo row of the CTA
// below (above), the slab's own ghost row beyond a wall (bc applied), or,
// on a level one CTA holds, its own opposite ghost row.
template <typename T>
struct Edge {
  T *lo, *hi;
  int lo_row, hi_row;
  bool lo_wall, hi_wall;
};
template <int DIM, typename T>
__device__ __forceinline__ Edge<T> edge_of(T* q, const Geo& g, const Part& pt, int lo_rows, const UniBC& bc) {
  Edge<T> E;
  E.lo_wall = bc.phys[DIM - 1] && pt.first;
  E.hi_wall = bc.phys[DIM - 1] && pt.last;
  E.lo = pt.shared && !E.lo_wall ? on_rank(q, pt.lo) : q;
  E.hi = pt.shared && !E.hi_wall ? on_rank(q, pt.hi) : q;
  E.lo_row = E.lo_wall ? 0 : (pt.shared ? lo_rows : g.nr) + 1;
  E.hi_row = E.hi_wall ? g.nr + 1 : 0;
  return E;
}

// The face images of cell (i, j, k) (local row last) of a slab, whose NV
// values are w.  Extents are at least 2; a slab may hold one row.
template <class TR, int DIM>
__device__ __forceinline__ void push_slab(typename TR::T* q, const Geo& g, const Edge<typename TR::T>& E, int i, int j,
                                          int k, const typename TR::T* w, const UniBC& bc,
                                          const typename TR::Par& par) {
  const int row = DIM == 2 ? j : k, st = DIM == 2 ? g.sy : g.sz;
  const int c = gcell<DIM>(g, i, j, k);
  if (i == 1 || i == g.n0) {
    const bool lo = i == 1;
    const int b = c + (bc.phys[0] ? (lo ? -1 : 1) : (lo ? g.n0 : -g.n0));
#pragma unroll
    for (int v = 0; v < TR::NV; v++)
      q[v * g.sq + b] = bc.phys[0] ? TR::wall(w[v], bc.mask, v) : TR::shift(w[v], lo ? 1 : 2, v, par);
  }
  if (DIM == 3 && (j == 1 || j == g.n1)) {
    const bool lo = j == 1;
    const int b = c + g.sy * (bc.phys[1] ? (lo ? -1 : 1) : (lo ? g.n1 : -g.n1));
#pragma unroll
    for (int v = 0; v < TR::NV; v++) q[v * g.sq + b] = bc.phys[1] ? TR::wall(w[v], bc.mask, v) : w[v];
  }
  if (row == 1) {
#pragma unroll
    for (int v = 0; v < TR::NV; v++)
      E.lo[v * g.sq + c + (E.lo_row - row) * st] = E.lo_wall ? TR::wall(w[v], bc.mask, v) : w[v];
  }
  if (row == g.nr) {
#pragma unroll
    for (int v = 0; v < TR::NV; v++)
      E.hi[v * g.sq + c + (E.hi_row - row) * st] = E.hi_wall ? TR::wall(w[v], bc.mask, v) : w[v];
  }
}

// The value at a cell of a slab's ghosted range whose edge and corner ghosts
// may be stale: columns and rows beyond a face from their interior cell, the
// offset across x before the walls as SetGhost applies them (a wall's ghost
// row, already through UserBC, would take the offset after it); the halo rows
// as they are
template <class TR, int DIM>
__device__ __forceinline__ typename TR::T slab_value(const typename TR::T* q, const Geo& g, const Part& pt, int i,
                                                     int j, int k, int v, const UniBC& bc,
                                                     const typename TR::Par& par) {
  int nb = 0, sh = 0, si = i, sj = j, sk = k;
  if (i < 1 || i > g.n0) {
    if (bc.phys[0]) {
      si = i < 1 ? 1 : g.n0;
      nb++;
    } else {
      si = i < 1 ? g.n0 : 1;
      sh = i < 1 ? 2 : 1;
    }
  }
  if (DIM == 3 && (j < 1 || j > g.n1)) {
    if (bc.phys[1]) {
      sj = j < 1 ? 1 : g.n1;
      nb++;
    } else {
      sj = j < 1 ? g.n1 : 1;
    }
  }
  int& row = DIM == 2 ? sj : sk;
  if (bc.phys[DIM - 1] && ((row < 1 && pt.first) || (row > g.nr && pt.last))) {
    row = row < 1 ? 1 : g.nr;
    nb++;
  }
  typename TR::T u = TR::shift(q[v * g.sq + gcell<DIM>(g, si, sj, sk)], sh, v, par);
#pragma unroll
  for (int z = 0; z < DIM; z++)
    if (z < nb) u = TR::wall(u, bc.mask, v);
  return u;
}

// This CTA's view of level x.  REMOTE: a level that CTA 0 holds alone is
// addressed in its shared memory by every CTA (else only CTA 0 may ask).
template <class TR, int DIM, bool REMOTE>
__device__ __forceinline__ View<typename TR::T> slab_view(const UniCycle& A, int x, int rank, Part& pt) {
  using T = typename TR::T;
  const UniLev& L = A.L[x];
  View<T> V;
  T* sm = reinterpret_cast<T*>(uni_smem);
  const int N = L.n[DIM - 1];
  int r0 = 0, nr = N;
  pt = Part{L.mul != 0, true, true, 0, 0, N};
  if (L.mul) {
    const UniRank& R = A.R[rank];
    r0 = R.row0 * L.mul;
    nr = R.rows * L.mul;
    pt.first = rank == 0;
    pt.last = rank + 1 == A.ctas;
    pt.lo = rank ? rank - 1 : A.ctas - 1;
    pt.hi = pt.last ? 0 : rank + 1;
    pt.lo_rows = A.R[pt.lo].rows * L.mul;
  } else if (REMOTE && rank) {
    sm = on_rank(sm, 0);
  }
  const int sy = L.n[0] + 2, sz = sy * (L.n[1] + 2), rows = L.maxr + 2;
  V.g = Geo{L.n[0], L.n[1], N, r0, nr, sy, sz, (DIM == 2 ? sy : sz) * rows};
  const int c0 = L.n[0] >> 1, c1 = L.n[1] >> 1, csy = c0 + 2, csz = csy * (c1 + 2);
  V.gc = Geo{c0, c1, N >> 1, r0 >> 1, nr >> 1, csy, csz, (DIM == 2 ? csy : csz) * ((L.maxr >> 1) + 2)};
  V.sf = L.n[0] * (DIM == 3 ? L.n[1] : 1) * L.maxr;
  V.q = sm + L.q;
  V.f = sm + L.f;
  V.c = sm + L.c;
  V.x = sm + L.x;
  V.d = &L.d;
  return V;
}

// The edge and corner images of this CTA's rows of a ghosted array, in its
// own ghosts and, of a shared level, in the neighbours' halo rows: one thread
// a cell of the shell, those beyond a single face left as push_slab wrote
// them.
template <class TR, int DIM>
__device__ __forceinline__ void images(typename TR::T* q, const Geo& g, const Part& pt, int lo_rows, const UniDiv& de0,
                                       const UniDiv& dring, int t0, int nt, const UniBC& bc,
                                       const typename TR::Par& par) {
  using T = typename TR::T;
  const int e0 = g.n0 + 2, cap = DIM == 3 ? e0 * (g.n1 + 2) : e0;
  const int ring = DIM == 3 ? 2 * e0 + 2 * g.n1 : 2;
  const int units = 2 * cap + g.nr * ring;
  for (int t = t0; t < units; t += nt) {
    // the image's cell: i, j in the ghosted range; `row` the source row, and
    // where the image goes
    int i, j = 0, row, to_row, nb = 0, sh = 0;
    T* dst = q;
    if (t < 2 * cap) {  // the first row (hi = 0) below itself, the last one above
      const int hi = t >= cap, u = t - hi * cap;
      if (DIM == 3) fdivmod(u, de0, j, i);
      else i = u;
      row = hi ? g.nr : 1;
      if (bc.phys[DIM - 1] && (hi ? pt.last : pt.first)) {
        to_row = hi ? g.nr + 1 : 0;
        nb = 1;
      } else if (pt.shared) {
        dst = on_rank(q, hi ? pt.hi : pt.lo);
        to_row = hi ? 0 : lo_rows + 1;
      } else {
        to_row = hi ? 0 : g.nr + 1;
      }
    } else {
      int u;
      if (DIM == 2) {
        u = t - 2 * cap;
        row = (u >> 1) + 1;
        i = (u & 1) ? g.n0 + 1 : 0;
      } else {
        fdivmod(t - 2 * cap, dring, row, u);
        row++;
        if (u < 2 * e0) {
          j = u < e0 ? 0 : g.n1 + 1;
          i = u < e0 ? u : u - e0;
        } else {
          j = ((u - 2 * e0) >> 1) + 1;
          i = (u & 1) ? g.n0 + 1 : 0;
        }
      }
      to_row = row;
    }
    int beyond = t < 2 * cap;
    auto src = [&](int x, int n, int d) {
      if (x >= 1 && x <= n) return x;
      beyond++;
      if (bc.phys[d]) {
        nb++;
        return x < 1 ? 1 : n;
      }
      if (d == 0) sh = x < 1 ? 2 : 1;
      return x < 1 ? n : 1;
    };
    const int si = src(i, g.n0, 0), sj = DIM == 3 ? src(j, g.n1, 1) : 0;
    if (beyond < 2) continue;
    const int a = DIM == 2 ? row * g.sy + si : row * g.sz + sj * g.sy + si;
    const int b = DIM == 2 ? to_row * g.sy + i : to_row * g.sz + j * g.sy + i;
#pragma unroll
    for (int v = 0; v < TR::NV; v++) {
      T u = TR::shift(q[v * g.sq + a], sh, v, par);
#pragma unroll
      for (int z = 0; z < DIM; z++)
        if (z < nb) u = TR::wall(u, bc.mask, v);
      dst[v * g.sq + b] = u;
    }
  }
}

// nsmooth relaxation passes of a slab (LevelRelax, afasroutines.f90:532-557):
// per colour the cells and their face images, then sync().  A thread keeps
// its cell of each colour when every cell has a thread.
template <class TR, int DIM, typename F>
__device__ __forceinline__ void smooth_slab(const View<typename TR::T>& V, const Part& pt, int nsmooth, bool coarsest,
                                            int t, int nt, const PatchDev& P, const UniBC& bc,
                                            const typename TR::Par& par, F&& sync) {
  const Geo& g = V.g;
  const int units = colour_units<DIM>(g);
  const Edge<typename TR::T> E = edge_of<DIM>(V.q, g, pt, pt.lo_rows, bc);
  auto cell = [&](int ipass, int i, int j, int k) {
    const int c = gcell<DIM>(g, i, j, k);
    TR::template relax<DIM>(V, c, icell<DIM>(g, i, j, k), ipass, P, par);
    typename TR::T w[TR::NV];
#pragma unroll
    for (int v = 0; v < TR::NV; v++) w[v] = V.q[v * g.sq + c];
    push_slab<TR, DIM>(V.q, g, E, i, j, k, w, bc, par);
  };
  if (units <= nt) {
    int i[2] = {0, 0}, j[2], k[2];
    bool on[2] = {false, false};
    if (t < units) {
      on[0] = colour_unit<DIM>(g, *V.d, t, 1, i[0], j[0], k[0]);
      on[1] = colour_unit<DIM>(g, *V.d, t, 2, i[1], j[1], k[1]);
    }
    for (int s = 0; s < nsmooth; s++) {
#pragma unroll 1
      for (int c = 0; c < 2; c++) {
        if (c ? on[1] : on[0])
          cell(TR::ipass(c + 1, coarsest), c ? i[1] : i[0], c ? j[1] : j[0], c ? k[1] : k[0]);
        sync();
      }
    }
    return;
  }
  for (int s = 0; s < 2 * nsmooth; s++) {
    const int c = 1 + (s & 1);
#pragma unroll 1
    for (int u = t; u < units; u += nt) {
      int i, j, k;
      if (colour_unit<DIM>(g, *V.d, u, c, i, j, k)) cell(TR::ipass(c, coarsest), i, j, k);
    }
    sync();
  }
}

// RestrictSolution of a slab with the face images of the coarse image and of
// the parent's q; EU: the parent's slab edges when it is shared out too
template <class TR, int DIM>
__device__ __forceinline__ void restrict_slab(const View<typename TR::T>& V, const View<typename TR::T>& U,
                                              const Part& pt, const Part& pu, int t, int nt, const UniBC& bc,
                                              const typename TR::Par& par) {
  using T = typename TR::T;
  const Geo &g = V.g, &gc = V.gc;
  const int units = inner_units<DIM>(gc);
  const int up = gc.r0 - U.g.r0;  // the parent's local row of the coarse image's row 0
  const Edge<T> E = edge_of<DIM>(V.c, gc, pt, pt.lo_rows >> 1, bc);
  const Edge<T> EU = edge_of<DIM>(U.q, U.g, pu, pu.lo_rows, bc);
  for (int u = t; u < units; u += nt) {
    int ci, cj, ck;
    inner_unit<DIM>(V.d->c0, V.d->c1, u, ci, cj, ck);
    const int f = gcell<DIM>(g, 2 * ci, 2 * cj, 2 * ck);
    const int pj = DIM == 2 ? cj + up : cj, pk = ck + up;
    T w[TR::NV];
#pragma unroll
    for (int v = 0; v < TR::NV; v++) {
      w[v] = mean<DIM>(V.q + v * g.sq + f, g.sy, g.sz);
      V.c[v * gc.sq + gcell<DIM>(gc, ci, cj, ck)] = w[v];
      U.q[v * U.g.sq + gcell<DIM>(U.g, ci, pj, pk)] = w[v];
    }
    push_slab<TR, DIM>(V.c, gc, E, ci, cj, ck, w, bc, par);
    push_slab<TR, DIM>(U.q, U.g, EU, ci, pj, pk, w, bc, par);
  }
}

// Residual of a slab, one thread a fine cell: r = f - Op(q) to the CTA's
// scratch (f's layout) and, FP64, to rf in global memory
template <class TR, int DIM>
__device__ __forceinline__ void resid_cells(const View<typename TR::T>& V, typename TR::T* r, typename TR::T* rf,
                                            int rf_sf, int t0, int nt, const PatchDev& P, const typename TR::Par& par) {
  using T = typename TR::T;
  const Geo& g = V.g;
  const int units = inner_units<DIM>(g);
  for (int t = t0; t < units; t += nt) {
    int i, j, k;
    inner_unit<DIM>(V.d->n0, V.d->n1, t, i, j, k);
    const int c = gcell<DIM>(g, i, j, k);
    T o[TR::NV];
    TR::template op<DIM>(V.q, c, g, V, c, t, P, par, o);
#pragma unroll
    for (int v = 0; v < TR::NV; v++) {
      const T e = V.f[v * V.sf + t] - o[v];
      r[v * V.sf + t] = e;
      if (TR::kStoreRf) rf[v * rf_sf + t] = e;
    }
  }
}
// CoarseLoadingFunction from that residual
template <class TR, int DIM>
__device__ __forceinline__ void load_cells(const View<typename TR::T>& V, const View<typename TR::T>& U,
                                           const typename TR::T* r, int t0, int nt, const PatchDev& PU,
                                           const typename TR::Par& par) {
  using T = typename TR::T;
  const Geo &g = V.g, &gc = V.gc;
  const int units = inner_units<DIM>(gc);
  const int up = gc.r0 - U.g.r0;
  for (int t = t0; t < units; t += nt) {
    int ci, cj, ck;
    inner_unit<DIM>(V.d->c0, V.d->c1, t, ci, cj, ck);
    const int pj = DIM == 2 ? cj + up : cj, pk = ck + up;
    const int fu = icell<DIM>(U.g, ci, pj, pk);
    T cr[TR::NV];
    TR::template op<DIM>(V.c, gcell<DIM>(gc, ci, cj, ck), gc, U, gcell<DIM>(U.g, ci, pj, pk), fu, PU, par, cr);
#pragma unroll
    for (int v = 0; v < TR::NV; v++)
      U.f[v * U.sf + fu] =
          mean<DIM>(r + v * V.sf + icell<DIM>(g, 2 * ci, 2 * cj, 2 * ck), g.n0, g.n0 * g.n1) + cr[v];
  }
}

// CorrectFine step 2 on a slab with the face images, one thread a fine cell
template <class TR, int DIM, bool INLINE_A>
__device__ __forceinline__ void correct_slab(const View<typename TR::T>& V, const View<typename TR::T>& U,
                                             const Part& pt, const Part& pu, int t, int nt, const UniBC& bc,
                                             const typename TR::Par& par) {
  using T = typename TR::T;
  const Geo &g = V.g, &gc = V.gc;
  const int units = inner_units<DIM>(g);
  const int up = gc.r0 - U.g.r0;
  const Edge<T> E = edge_of<DIM>(V.q, g, pt, pt.lo_rows, bc);
  for (int u = t; u < units; u += nt) {
    int i, j, k;
    inner_unit<DIM>(V.d->n0, V.d->n1, u, i, j, k);
    const int ci = i >> 1, cj = j >> 1, ck = DIM == 3 ? k >> 1 : 0;
    const bool fx = i & 1, fy = j & 1, fz = DIM == 3 && (k & 1);
    const int c = gcell<DIM>(g, i, j, k);
    T w[TR::NV];
#pragma unroll
    for (int v = 0; v < TR::NV; v++) {
      auto at = [&](int ii, int jj, int kk) -> T {
        if (!INLINE_A) return V.c[v * gc.sq + gcell<DIM>(gc, ii, jj, kk)];
        return slab_value<TR, DIM>(U.q, U.g, pu, ii, DIM == 2 ? jj + up : jj, kk + up, v, bc, par) -
               slab_value<TR, DIM>(V.c, gc, pt, ii, jj, kk, v, bc, par);
      };
      auto row = [&](int jj, int kk) -> T {  // the x stage at coarse row (jj, kk)
        const T lo = at(ci, jj, kk), hi = at(ci + 1, jj, kk);
        return fx ? lo + triple<DIM>(hi) : triple<DIM>(lo) + hi;
      };
      auto plane = [&](int kk) -> T {
        const T lo = row(cj, kk), hi = row(cj + 1, kk);
        return fy ? lo + triple<DIM>(hi) : triple<DIM>(lo) + hi;
      };
      T add;
      if (DIM == 2) {
        add = scaled<-4>(plane(0));
      } else {
        const T lo = plane(ck), hi = plane(ck + 1);
        add = scaled<-6>(fz ? lo + triple<DIM>(hi) : triple<DIM>(lo) + hi);
      }
      w[v] = V.q[v * g.sq + c] + add;
      V.q[v * g.sq + c] = w[v];
    }
    push_slab<TR, DIM>(V.q, g, E, i, j, k, w, bc, par);
  }
}

// rows lo .. hi of a ghosted array of nv variables between the slab (local
// rows) and global memory (row r0 + local row): up != 0 stores
template <typename T, int DIM>
__device__ __forceinline__ void copy_rows(T* s, const Geo& g, T* gl, long long gsq, int nv, int lo, int hi, bool up) {
  const int e0 = g.n0 + 2, plane = DIM == 2 ? e0 : e0 * (g.n1 + 2);
  const int n = plane * (hi - lo + 1);
  for (int v = 0; v < nv; v++) {
    T* a = s + v * g.sq + lo * plane;
    T* b = gl + v * gsq + (long long)(g.r0 + lo) * plane;
    if (up)
      for (int t = threadIdx.x; t < n; t += blockDim.x) b[t] = a[t];
    else
      for (int t = threadIdx.x; t < n; t += blockDim.x) a[t] = b[t];
  }
}
// the slab's rows of an interior array of nv variables
template <typename T, int DIM>
__device__ __forceinline__ void copy_inner(T* s, const Geo& g, int sf, T* gl, long long gsf, int nv, bool up) {
  const int plane = DIM == 2 ? g.n0 : g.n0 * g.n1;
  const int n = plane * g.nr;
  for (int v = 0; v < nv; v++) {
    T* a = s + v * sf;
    T* b = gl + v * gsf + (long long)g.r0 * plane;
    if (up)
      for (int t = threadIdx.x; t < n; t += blockDim.x) b[t] = a[t];
    else
      for (int t = threadIdx.x; t < n; t += blockDim.x) a[t] = b[t];
  }
}

template <class TR, int DIM>
__global__ void __launch_bounds__(kUniThreads, 1) k_uni_cycle(const PatchDev* __restrict__ P, typename TR::Mem m,
                                                              const __grid_constant__ UniCycle A,
                                                              typename TR::Par par) {
  after_previous();
  using T = typename TR::T;
  const int rank = A.ctas > 1 ? my_rank() : 0;
  const int t = threadIdx.x, nt = blockDim.x;
  __shared__ __align__(16) PatchDev sp[kNLev];
  stage_table(sp, P, A);
  auto all = [&] {
    if (A.ctas > 1) cluster_sync();
    else __syncthreads();
  };
  // a phase's end: the cluster's barrier on a shared level, the CTA's on CTA 0's own
  auto sync = [&](int x) {
    if (A.L[x].mul) all();
    else __syncthreads();
  };
  TR::template stage_in<DIM>(A, rank, sp, m);
  all();
  Part pt, pu;
  auto smooth = [&](int x) {
    const View<T> V = slab_view<TR, DIM, false>(A, x, rank, pt);
    smooth_slab<TR, DIM>(V, pt, A.nsmooth, x == A.nl - 1, t, nt, sp[x], A.bc, par, [&] { sync(x); });
  };
  T* const scratch = reinterpret_cast<T*>(uni_smem) + A.scratch;
  // down: the levels shared out, then CTA 0 alone
  for (int x = 0; x < A.nl; x++) {
    if (!A.L[x].mul && rank) break;
    smooth(x);
    if (x + 1 == A.nl) break;
    const View<T> V = slab_view<TR, DIM, false>(A, x, rank, pt), U = slab_view<TR, DIM, true>(A, x + 1, rank, pu);
    restrict_slab<TR, DIM>(V, U, pt, pu, t, nt, A.bc, par);
    // rf, and the residual the coarse loading averages
    T* rf = TR::rf(sp[x], m);
    if (TR::kStoreRf) rf += V.g.r0 * V.g.n0 * (DIM == 3 ? V.g.n1 : 1);
    resid_cells<TR, DIM>(V, scratch, rf, (int)sp[x].sf, t, nt, sp[x], par);
    sync(x);
    load_cells<TR, DIM>(V, U, scratch, t, nt, sp[x + 1], par);
    // the image's edges and corners, which CorrectFine's first step reads
    if (TR::kStoreRf) images<TR, DIM>(V.c, V.gc, pt, pt.lo_rows >> 1, V.d->ce0, V.d->cring, t, nt, A.bc, par);
    // the next level's smoothing reads f where this CTA wrote it, unless CTA 0 takes the level over
    if (pt.shared && !pu.shared) all();
    else __syncthreads();
  }
  // up
  for (int x = A.nl - 2; x >= 0; x--) {
    if (!A.L[x].mul && rank) continue;
    if (A.L[x].mul && !A.L[x + 1].mul) all();  // CTA 0 has finished the levels it holds
    const View<T> V = slab_view<TR, DIM, false>(A, x, rank, pt), U = slab_view<TR, DIM, true>(A, x + 1, rank, pu);
    if (TR::kStoreRf) {
      correct_a<TR, DIM, false>(V, U, pu, t, nt, A.bc, par);
      __syncthreads();
    }
    correct_slab<TR, DIM, !TR::kStoreRf>(V, U, pt, pu, t, nt, A.bc, par);
    sync(x);
    smooth(x);
  }
  // edges and corners of what leaves
  for (int x = 0; x < (TR::kStoreRf ? A.nl : 1); x++) {
    if (!A.L[x].mul && rank) break;
    const View<T> V = slab_view<TR, DIM, false>(A, x, rank, pt);
    images<TR, DIM>(V.q, V.g, pt, pt.lo_rows, V.d->e0, V.d->ring, t, nt, A.bc, par);
  }
  all();
  TR::template stage_out<DIM>(A, rank, sp, m);
  // a CTA's shared memory stays while another may still address it
  all();
}

// ---- launchers ----

template <class TR>
struct UniLaunchers {
  using Mem = typename TR::Mem;
  using Par = typename TR::Par;
  static int blocks(long long units) { return (int)((units + kBlock - 1) / kBlock); }
  static long long cells(const int* n) { return (long long)n[0] * n[1] * n[2]; }

  static int relax(const LaunchCtx& c, const UniBC& bc, int patch, const PatchDev& hp, int ipass,
                   int full) {
    const UniPatch p = uni_patch_of(hp);
    const int nb = blocks((long long)((hp.mx[0] + 1) / 2) * hp.mx[1] * hp.mx[2]);
    if (c.ndims == 2)
      launch_after(k_uni_relax<TR, 2>, nb, kBlock, 0, c.s, c.P, TR::mem(c), patch, p, ipass, full, bc, TR::par(c));
    else
      launch_after(k_uni_relax<TR, 3>, nb, kBlock, 0, c.s, c.P, TR::mem(c), patch, p, ipass, full, bc, TR::par(c));
    return 1;
  }
  static int restrict_load(const LaunchCtx& c, const UniBC& bc, int patch, const PatchDev& hp, const PatchDev& hu) {
    const UniPatch p = uni_patch_of(hp), u = uni_patch_of(hu);
    const int nb = blocks(cells(hp.cmx));
    if (c.ndims == 2) {
      launch_after(k_uni_restrict<TR, 2>, nb, kBlock, 0, c.s, TR::mem(c), p, u, bc, TR::par(c));
      launch_after(k_uni_load<TR, 2>, nb, kBlock, 0, c.s, c.P, TR::mem(c), patch, p, hp.parent, u, TR::par(c));
    } else {
      launch_after(k_uni_restrict<TR, 3>, nb, kBlock, 0, c.s, TR::mem(c), p, u, bc, TR::par(c));
      launch_after(k_uni_load<TR, 3>, nb, kBlock, 0, c.s, c.P, TR::mem(c), patch, p, hp.parent, u, TR::par(c));
    }
    return 2;
  }
  static int correct(const LaunchCtx& c, const UniBC& bc, const PatchDev& hp, const PatchDev& hu) {
    const UniPatch p = uni_patch_of(hp), u = uni_patch_of(hu);
    int n = 1;
    if (TR::kStoreRf) {
      const int na = blocks(cells(hp.cn));
      if (c.ndims == 2) launch_after(k_uni_correct_a<TR, 2>, na, kBlock, 0, c.s, TR::mem(c), p, u, bc, TR::par(c));
      else launch_after(k_uni_correct_a<TR, 3>, na, kBlock, 0, c.s, TR::mem(c), p, u, bc, TR::par(c));
      n++;
    }
    const int nb = blocks((long long)(hp.cmx[0] + 1) * (hp.cmx[1] + 1) * (c.ndims == 3 ? hp.cmx[2] + 1 : 1));
    if (c.ndims == 2) launch_after(k_uni_correct_b<TR, 2>, nb, kBlock, 0, c.s, TR::mem(c), p, u, bc, TR::par(c));
    else launch_after(k_uni_correct_b<TR, 3>, nb, kBlock, 0, c.s, TR::mem(c), p, u, bc, TR::par(c));
    return n;
  }
  static int ghost(const LaunchCtx& c, const UniBC& bc, const PatchDev& hp) {
    const UniPatch p = uni_patch_of(hp);
    const int nb = blocks(cells(hp.qn) - cells(hp.mx));
    if (c.ndims == 2) launch_after(k_uni_ghost<TR, 2>, nb, kBlock, 0, c.s, TR::mem(c), p, bc, TR::par(c));
    else launch_after(k_uni_ghost<TR, 3>, nb, kBlock, 0, c.s, TR::mem(c), p, bc, TR::par(c));
    return 1;
  }
  static int walls(const LaunchCtx& c, const UniBC& bc, const PatchDev& hp) {
    if (!bc.phys[0] && !bc.phys[1] && !(c.ndims == 3 && bc.phys[2])) return 0;
    const UniPatch p = uni_patch_of(hp);
    const int nb = blocks(cells(hp.qn) - cells(hp.mx));
    if (c.ndims == 2) launch_after(k_uni_walls<TR, 2>, nb, kBlock, 0, c.s, TR::mem(c), p, bc, TR::par(c));
    else launch_after(k_uni_walls<TR, 3>, nb, kBlock, 0, c.s, TR::mem(c), p, bc, TR::par(c));
    return 1;
  }
  static int fill(const LaunchCtx& c, const UniBC& bc, const PatchDev& hp, const PatchDev& hu, int fields) {
    const UniPatch p = uni_patch_of(hp), u = uni_patch_of(hu);
    const int nb = blocks(cells(hp.cmx));
    if (c.ndims == 2) launch_after(k_uni_fill<TR, 2>, nb, kBlock, 0, c.s, TR::mem(c), p, u, fields, bc, TR::par(c));
    else launch_after(k_uni_fill<TR, 3>, nb, kBlock, 0, c.s, TR::mem(c), p, u, fields, bc, TR::par(c));
    return 1;
  }
  static int fill_small(const LaunchCtx& c, const UniCycle& A, int fields) {
    if (c.ndims == 2)
      launch_after(k_uni_fill_small<TR, 2>, 1, kUniFillThreads, 0, c.s, c.P, TR::mem(c), A, fields, TR::par(c));
    else
      launch_after(k_uni_fill_small<TR, 3>, 1, kUniFillThreads, 0, c.s, c.P, TR::mem(c), A, fields, TR::par(c));
    return 1;
  }
  static int cycle(const LaunchCtx& c, const UniCycle& A, int smem) {
    auto k = c.ndims == 2 ? k_uni_cycle<TR, 2> : k_uni_cycle<TR, 3>;
    cudaError_t e = launch_cluster(k, A.ctas, A.threads, smem, c.s, c.P, TR::mem(c), A, TR::par(c));
    return e == cudaSuccess ? 1 : -1;
  }
  // raise the kernel's limits (clusters above the portable 8 CTAs, dynamic
  // shared memory) and report how many clusters of `ctas` fit at once
  static int cycle_fit(int ndims, int ctas, int smem) {
    auto fit = [&](auto k) {
      if (cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) return 0;
      if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kUniSmemMax) != cudaSuccess) return 0;
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(ctas);
      cfg.blockDim = dim3(kUniThreads);
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
    const int n = ndims == 2 ? fit(k_uni_cycle<TR, 2>) : fit(k_uni_cycle<TR, 3>);
    cudaGetLastError();  // a shape that does not fit is an answer, not an error
    return n;
  }
  static PluginUni table() {
    return PluginUni{TR::NV, TR::kXPlanes, TR::kXGhosted, (int)sizeof(typename TR::T), &relax, &restrict_load, &correct,
                     &ghost, &walls, &fill, &fill_small, &cycle, &cycle_fit};
  }
};

}  // namespace uni
}  // namespace bsamg
