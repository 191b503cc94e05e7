#include "uni.h"

#include <algorithm>

namespace bsamg {

bool uni_eligible(const Hier& H) {
  if (H.mbc != 1 || !find_plugin(H.problem)->face_stencils) return false;
  const HostPatch* root = nullptr;
  for (int l = 0; l >= H.minlevel; l--) {
    if (H.L(l).patches.size() != 1) return false;
    const HostPatch& P = H.patches[H.L(l).patches[0]];
    if (!root) root = &P;
    for (int d = 0; d < H.ndims; d++) {
      const int a = P.mthbc[2 * d], b = P.mthbc[2 * d + 1];
      if (a != b || (a != 2 && a != 10) || a != root->mthbc[2 * d]) return false;
      if (a == 2 && (!H.periodic || P.mx[d] % 2)) return false;  // odd: two cells of one colour are neighbours
      if (l > H.minlevel) {
        const HostPatch& Q = H.patches[P.parent];
        if (P.mbounds[d][0] != 1 || P.mbounds[d][1] != Q.mx[d] || P.cmx[d] != Q.mx[d] || P.mx[d] != 2 * Q.mx[d])
          return false;
      }
    }
    // the kernels index a level's variables with 32-bit offsets
    long long sq = 1;
    for (int d = 0; d < H.ndims; d++) {
      if (P.mx[d] < 2) return false;  // a cell between two faces has two images
      sq *= P.mx[d] + 2;
    }
    if (sq * H.nrvars >= (1LL << 31)) return false;
  }
  return true;
}

UniBC uni_bc(const Hier& H) {
  UniBC b{};
  const HostPatch& P = H.patches[H.L(0).patches[0]];
  for (int d = 0; d < H.ndims; d++) b.phys[d] = P.mthbc[2 * d] == 10;
  b.mask = find_plugin(H.problem)->bc_mask(H.ndims);
  return b;
}

namespace {

// Largest level the cluster takes over.  FP64: 16 SMs issue 32 FP64
// operations a clock, so a colour sweep of 4096 cells costs about 1.2 us of
// pipe time and one of 16384 cells 5 us, where a launch over the whole GPU
// costs about 2.5 us whatever the size.  FP32 sweeps are latency-bound to the
// size the shared memory holds.
long long cycle_cells(const PluginUni& U) { return U.elem == 8 ? 6144 : 40960; }

// Time of one colour sweep (us) of a level of `cells` on `ctas` SMs: the
// barrier and latency of the phase plus the pipe (FP64: 2 operations a clock
// and SM, about 20 per cell and variable; FP32: about 64 issue slots a clock
// for 100 instructions per cell).
double sweep_us(const PluginUni& U, long long cells, int ctas, bool shared) {
  const double per = U.elem == 8 ? 10.0 * U.nv : 0.8 * U.nv;
  return (shared ? 0.55 : 0.35) + 0.5 * (double)cells * per / ctas / 2000.0;
}

// Plan with the first `share` levels shared out; false when it does not fit
bool lay_out(const Hier& H, const PluginUni& U, int top, int minlevel, int share, UniCycle& A, int* smem) {
  const int D = H.ndims, slow = D - 1;
  A.nl = top - minlevel + 1;
  auto patch = [&](int x) -> const HostPatch& { return H.patches[H.L(top - x).patches[0]]; };
  int nc = 1;
  A.ctas = 1;
  if (share) {
    // the partition follows the rows of the first solo level (each CTA
    // restricts whole coarse rows), or of the last level when all are shared
    nc = patch(std::min(share, A.nl - 1)).mx[slow];
    A.ctas = std::min(16, nc);
    if (A.ctas < 2) return false;
  }
  int most = 0;
  for (int r = 0; r < A.ctas; r++) {
    const int a = r * nc / A.ctas, b = (r + 1) * nc / A.ctas;
    A.R[r] = UniRank{(short)a, (short)(b - a)};
    most = std::max(most, b - a);
  }
  long long o = 0, scratch = 0;
  auto add = [&](long long n) {
    const long long at = o;
    o += (n + 3) & ~3LL;
    return (int)at;
  };
  for (int x = 0; x < A.nl; x++) {
    const HostPatch& P = patch(x);
    UniLev& L = A.L[x];
    L.patch = H.L(top - x).patches[0];
    for (int d = 0; d < 3; d++) L.n[d] = P.mx[d];
    L.mul = x < share ? 1 << (std::min(share, A.nl - 1) - x) : 0;
    L.maxr = L.mul ? most * L.mul : P.mx[slow];
    L.d = uni_dim(P.mx);
    const long long plane = (long long)(P.mx[0] + 2) * (D == 3 ? P.mx[1] + 2 : 1) * (L.maxr + 2);
    const long long inner = (long long)P.mx[0] * (D == 3 ? P.mx[1] : 1) * L.maxr;
    const long long cplane = (long long)(P.mx[0] / 2 + 2) * (D == 3 ? P.mx[1] / 2 + 2 : 1) * (L.maxr / 2 + 2);
    L.q = add(U.nv * plane);
    L.f = add(U.nv * inner);
    L.c = x + 1 < A.nl ? add(U.nv * cplane) : 0;
    L.x = add(U.nx * (U.x_ghosted ? plane : inner));
    if (x + 1 < A.nl) scratch = std::max(scratch, U.nv * inner);
    if (o * U.elem > kUniSmemMax) return false;
  }
  A.scratch = add(scratch);
  if (o * U.elem > kUniSmemMax) return false;
  *smem = (int)(o * U.elem);
  return true;
}

}  // namespace

const Hier::UniPlan* uni_plan(Hier& H, const PluginUni& U, int level, int minlevel, int nsmooth) {
  if (!H.uni || H.tail_cells == 0 || level > 0) return nullptr;
  auto key = std::make_tuple(level, minlevel, nsmooth, U.elem);
  auto it = H.uni_plans.find(key);
  if (it == H.uni_plans.end()) {
    Hier::UniPlan best{};
    auto cells = [&](int l) {
      const HostPatch& P = H.patches[H.L(l).patches[0]];
      return (long long)P.mx[0] * P.mx[1] * P.mx[2];
    };
    for (int top = level; top >= minlevel && best.A.nl == 0; top--) {
      if (cells(top) > cycle_cells(U)) continue;
      double best_us = 0.0;
      for (int share = 0; share <= top - minlevel + 1; share++) {
        UniCycle A{};
        int smem = 0;
        if (!lay_out(H, U, top, minlevel, share, A, &smem)) continue;
        if (U.cycle_fit(H.ndims, A.ctas, smem) < 1) continue;
        double us = 0.0;
        for (int x = 0; x < A.nl; x++)
          us += sweep_us(U, cells(top - x), x < share ? A.ctas : 1, x < share) + (x == share && share ? 0.5 : 0.0);
        if (best.A.nl && us >= best_us) continue;
        best_us = us;
        best.A = A;
        best.smem = smem;
        best.top = top;
      }
    }
    if (best.A.nl) {
      best.A.nsmooth = nsmooth;
      best.A.bc = H.ubc;
      // one thread a cell of a colour, in whole warps
      long long units = cells(best.top) / 2 / best.A.ctas;
      best.A.threads = units > 256 ? kUniThreads : 256;
    }
    it = H.uni_plans.emplace(key, best).first;
  }
  return it->second.A.nl ? &it->second : nullptr;
}

// Levels from which one CTA does the rest of FillDown: above, a launch a level
// over the GPU is quicker.  The solves wait for it before they return (a step
// of five V-cycles with the line at 16384 | 8192 | 4096 | 1024 cells: 128^2 FP64
// 877 | 859 | 860 | 856 us, mixed 307 | 296 | 297 | 296, 128x64 FP64 784 | 784 |
// 776 | 776, growth 24^3 mixed 937 | 839 | 839 | 844; a fill of q at 32^3 25.0 |
// 25.0 | 25.1 | 24.0).
constexpr long long kFillSmallCells = 4096;

int uni_enq_fill(Hier& H, const PluginUni& U, int fields, int level, int minlevel) {
  const LaunchCtx c = H.lc();
  for (int l = level; l > minlevel; l--) {
    const int p = uni_patch(H, l);
    const HostPatch& P = H.patches[p];
    if ((long long)P.mx[0] * P.mx[1] * P.mx[2] <= kFillSmallCells && l - minlevel < kNLev) {  // the rest in one CTA
      UniCycle A{};
      A.bc = H.ubc;
      for (int x = l; x >= minlevel; x--) {
        A.L[A.nl].patch = uni_patch(H, x);
        A.L[A.nl++].d = uni_dim(H.hP[uni_patch(H, x)].mx);
      }
      return after_launch(H, U.fill_small(c, A, fields));
    }
    if (int r = after_launch(H, U.fill(c, H.ubc, H.hP[p], H.hP[uni_patch(H, l - 1)], fields))) return r;
  }
  return BSAMG_OK;
}

}  // namespace bsamg
