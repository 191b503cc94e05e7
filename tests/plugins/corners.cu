// A test-only problem whose operator reads the diagonal neighbours: one
// implicit Euler step of two uncoupled equations with a mixed derivative,
// u - c Lap(u) - d u_xy = u_old, relaxed pointwise on the Laplacian part.  FP64 only.
#include "plugin_def.cuh"

namespace bsamg {

struct Corners {
  static constexpr int kKind = 41;
  static constexpr const char* kName = "corners";
  static constexpr int kNV = 2;
  static constexpr int kNParams = 2;  // dt, strength of the mixed derivative
  static constexpr bool kCoeffsOnly = true;
  static constexpr bool kBox = false;
  static constexpr bool kMixed = false;

  static void set_params(ProbParams& pp, const double* prm, int) {
    pp.dt = prm[0];
    pp.user[0] = prm[1];
  }
  static void coefficients(const ProbParams& pp, int ndims, double h, double* c) {
    c[0] = pp.dt / (h * h);
    c[1] = 0.25 * pp.user[0] * pp.dt / (h * h);
    c[2] = 1.0 + 2.0 * ndims * c[0];
    c[3] = 0.0;
  }
  static int bc_mask(int) { return 1 | (2 << 8); }  // 2 - q, -q
  static int stats(int) { return 1; }

  __device__ __forceinline__ static double uxy(const double* a, long long c, long long sy) {
    return a[c + sy + 1] - a[c + sy - 1] - a[c - sy + 1] + a[c - sy - 1];
  }
  template <int DIM>
  __device__ __forceinline__ static void relax(const Cell64& x, const double* cf, const ProbParams&) {
    for (int v = 0; v < 2; v++) {
      double* u = x.q + v * x.sq;
      double s = u[x.c - 1] + u[x.c + 1] + u[x.c - x.sy] + u[x.c + x.sy];
      if (DIM == 3) s = s + u[x.c - x.sz] + u[x.c + x.sz];
      u[x.c] = (x.f[v * x.sf + x.fc] + cf[0] * s) / cf[2];
    }
  }
  template <int DIM>
  __device__ __forceinline__ static void op(const double* a, long long c, long long sy, long long sz, long long ps,
                                            const QoldView&, const double* cf, const ProbParams&, double* r) {
    for (int v = 0; v < 2; v++) {
      const double* u = a + v * ps;
      r[v] = u[c] - cf[0] * ulap<DIM>(u, c, sy, sz) - cf[1] * uxy(u, c, sy);
    }
  }
  template <int DIM>
  __device__ __forceinline__ static void source(const double*, long long, long long, long long, long long,
                                                const QoldView& qo, const double*, const ProbParams&, double* s) {
    s[0] = qo.p[0];
    s[1] = qo.p[qo.sq];
  }
  template <int DIM>
  __device__ __forceinline__ static void source_update(const double*, long long, long long, long long, long long,
                                                       const QoldView&, const double*, const ProbParams&,
                                                       double* su) {
    su[0] = 0.0;
    su[1] = 0.0;
  }
};

BSAMG_PLUGIN(Corners)

}  // namespace bsamg
