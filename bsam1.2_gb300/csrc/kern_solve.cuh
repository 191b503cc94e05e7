// The mixed-precision solve of an adaptive hierarchy in one launch of one
// thread-block cluster (included by kern_mixed.cuh; templates over the
// plugin struct).
//
// On an adaptive mesh every level is small (a few thousand cells on patches
// of 8-64 cells per side) and a V-cycle is a chain of some 300 dependent
// operations: colour sweeps, ghost programs, restriction, the FAS loading,
// prolongation.  As separate launches each costs a launch and a drain of the
// whole GPU for microseconds of work.  Here the host records the solve once
// per mesh as a program of phases over the same device work lists, and one
// cluster of up to 16 CTAs executes it: every phase is spread over all
// threads of the cluster and phases are separated by the cluster's hardware
// barrier (barrier.cluster arrive.release / wait.acquire, which orders the
// global-memory writes of one phase before the reads of the next for every
// thread of the cluster, about 0.25 us on GB300).  The coarse end of the
// V-cycle runs in CTA 0 alone, with CTA barriers, while the other CTAs wait.
// The loop of MultigridIterations (afasroutines.f90:78-104) runs on the
// device too: each outer iteration ends with the FP64 residual norm of the
// finest level, reduced in the same order as launch_norm_finish, and CTA 0
// records it and decides whether to stop (norm below the tolerance, a
// non-finite norm, or the last allowed V-cycle).  The host reads one control
// block after the launch.
//
// Every unit computes what the stand-alone kernel of the same operation
// computes, in the same order, so a solve gives bit for bit the iterates of
// the per-launch mixed path.  FP64 ghost programs and FillDown are written
// with explicitly rounded products and sums (this file is compiled with
// contraction on, the FP64 path's kernels without it).
#pragma once
#include <cuda_runtime.h>

namespace bsamg {
namespace mx {

__device__ __forceinline__ unsigned cluster_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ unsigned cluster_ctas() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
// every thread of every CTA of the cluster; the release/acquire pair makes
// all memory writes before it visible to all threads of the cluster after it
__device__ __forceinline__ void cluster_barrier() {
  __syncwarp();  // the aligned forms want the warp converged
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// the 256 threads of group g of this CTA (hardware barrier 1 + g)
__device__ __forceinline__ void group_barrier(int g) { asm volatile("bar.sync %0, 256;" ::"r"(1 + g) : "memory"); }

// C/F interpolation weights, LIBRARY/boundary.f90:54-63
constexpr double dA1 = -01.0 / 05.0, dA2 = 02.0 / 03.0, dA3 = 08.0 / 15.0;
constexpr double dB1 = 05.0 / 32.0, dB2 = 15.0 / 16.0, dB3 = -03.0 / 32.0;
constexpr double dC1 = 09.0 / 16.0, dC2 = 03.0 / 16.0, dC3 = 03.0 / 16.0, dC4 = 01.0 / 16.0;

// An FP64 ghost operation (the FP64 path's ghost_apply), each product and
// sum rounded on its own in the same order.  The variable loop has the
// plugin's constant bound: a runtime index into pp.qpo would place the
// parameters in local memory, which every cluster barrier evicts from L1.
template <int NV>
__device__ __forceinline__ void s_ghost64(const PatchDev* __restrict__ P, double* pool, const GhostOp& g,
                                          const ProbParams& pp) {
  const PatchDev& d = P[g.dp];
  const PatchDev& s = P[g.sp];
  double val[NV];  // every variable's loads before the first store
#pragma unroll
  for (int v = 0; v < NV; v++) {
    const double* dq = pool + d.oq + v * d.sq;
    const double* sq = pool + s.oq + v * s.sq;
    switch (g.type) {
      case kGCopy: val[v] = sq[g.s0]; break;
      case kGCopyAdd: val[v] = __dadd_rn(sq[g.s0], pp.qpo[v]); break;
      case kGCopySub: val[v] = __dsub_rn(sq[g.s0], pp.qpo[v]); break;
      case kGBC:
        val[v] = ((g.mask >> v) & 1) ? __dsub_rn(2.0, sq[g.s0]) : (((g.mask >> (8 + v)) & 1) ? -sq[g.s0] : sq[g.s0]);
        break;
      case kGCfA:
        val[v] = __dadd_rn(__dadd_rn(__dmul_rn(dA1, dq[g.s0]), __dmul_rn(dA2, dq[g.s1])), __dmul_rn(dA3, sq[g.c0]));
        break;
      case kGCfAB: {
        double c = __dadd_rn(__dadd_rn(__dmul_rn(dB1, sq[g.c0]), __dmul_rn(dB2, sq[g.c1])), __dmul_rn(dB3, sq[g.c2]));
        val[v] = __dadd_rn(__dadd_rn(__dmul_rn(dA1, dq[g.s0]), __dmul_rn(dA2, dq[g.s1])), __dmul_rn(dA3, c));
        break;
      }
      default: {
        double c = __dadd_rn(__dadd_rn(__dadd_rn(__dmul_rn(dC1, sq[g.c0]), __dmul_rn(dC2, sq[g.c1])),
                                       __dmul_rn(dC3, sq[g.c2])),
                             __dmul_rn(dC4, sq[g.c3]));
        val[v] = __dadd_rn(__dadd_rn(__dmul_rn(dA1, dq[g.s0]), __dmul_rn(dA2, dq[g.s1])), __dmul_rn(dA3, c));
        break;
      }
    }
  }
#pragma unroll
  for (int v = 0; v < NV; v++) pool[d.oq + v * d.sq + g.dcell] = val[v];
}

// Ghost images on a uniform level (kern_uni.cuh push): the FP64 solution's
// values, each rounding explicit as in s_ghost64; the correction's with the
// homogeneous conditions
template <int NVARS>
struct Push64 {
  using T = double;
  using Par = ProbParams;
  static constexpr int NV = NVARS;
  __device__ __forceinline__ static double shift(double w, int s, int v, const Par& pp) {
    return s == 0 ? w : (s == 1 ? __dadd_rn(w, pp.qpo[v]) : __dsub_rn(w, pp.qpo[v]));
  }
  __device__ __forceinline__ static double wall(double u, int mask, int v) {
    return ((mask >> v) & 1) ? __dsub_rn(2.0, u) : (((mask >> (8 + v)) & 1) ? -u : u);
  }
};
template <int NVARS>
struct Push32 {
  using T = float;
  using Par = int;
  static constexpr int NV = NVARS;
  __device__ __forceinline__ static float shift(float w, int, int, int) { return w; }
  __device__ __forceinline__ static float wall(float u, int mask, int v) { return ((mask >> v) & 0x101) ? -u : u; }
};
template <class TR, int DIM>
__device__ __forceinline__ void s_push(typename TR::T* base, const PatchDev& p, int i, int j, int k,
                                       const typename TR::T* w, const UniBC& bc, const typename TR::Par& par) {
  const int N = DIM == 3 ? p.mx[2] : p.mx[1];
  const uni::Geo g{p.mx[0], p.mx[1], N, 0, N, p.qn[0], p.qn[0] * p.qn[1], (int)p.sq};
  uni::push<TR, DIM>(base, g, i, j, k, w, true, bc, par);
}

// The operations of a uniform level that write their cells' images
// (kPushGhosts).  Its ghost program is two stages of a few hundred cells, on
// the critical path of every sweep: 6700 cycles on a 64^2 level, 3000 in the
// CTA that runs the coarse end alone.  (The prolongation sets four to eight
// cells a thread: its images are a phase of their own, kSUniGhost.)
template <class PL, int DIM>
__device__ __forceinline__ void s_relax_push(const PatchDev* __restrict__ P, float* fpool, const Blk b, int tid,
                                             int arg, const MxParams& mp, const UniBC& bc) {
  constexpr int NV = PL::kNV;
  const PatchDev& p = P[b.patch];
  int i, j, k;
  if (!color_cell<DIM>(p, b.start + tid, arg & 3, i, j, k)) return;
  const Cell32 x = cell32<PL, DIM, true>(p, fpool, i, j, k);
  if (arg & kRelax64) PL::template mx_relax<DIM, double>(x, p.c, mp);
  else PL::template mx_relax<DIM, float>(x, p.cf, mp);
  float w[NV];
  for (int v = 0; v < NV; v++) w[v] = x.e[v * x.sq + x.c];
  s_push<Push32<NV>, DIM>(x.e, p, i, j, k, w, bc, 0);
}
// u_restrict onto a uniform parent
template <int NV, int DIM>
__device__ __forceinline__ void s_restrict_push(const PatchDev* __restrict__ P, float* fpool, const Blk b, int tid,
                                                const UniBC& bc) {
  const PatchDev& p = P[b.patch];
  int ci, cj, ck;
  if (!interior_cell<DIM>(p.cmx, b.start + tid, ci, cj, ck)) return;
  const PatchDev& par = P[p.parent];
  float* fp = fbase<true>(fpool, p);
  float* fq = fbase<true>(fpool, par);
  const int pi = p.mb[0] + ci - 1, pj = p.mb[1] + cj - 1, pk = DIM == 3 ? p.mb[2] + ck - 1 : 1;
  float w[NV];
  for (int v = 0; v < NV; v++) {
    const float* e = fp + p.eq + v * p.sq;
    auto at = [&](int i, int j, int k) { return e[gofs<DIM>(p.qn, i, j, k)]; };
    w[v] = restrict_at32<DIM>(at, ci, cj, ck);
  }
  for (int v = 0; v < NV; v++) {
    fp[p.ecq + v * p.sc + gofs<DIM>(p.cn, ci, cj, ck)] = w[v];
    fq[par.eq + v * par.sq + gofs<DIM>(par.qn, pi, pj, DIM == 3 ? pk : 0)] = w[v];
  }
  s_push<Push32<NV>, DIM>(fq + par.eq, par, pi, pj, pk, w, bc, 0);
}

// FillDownLevel of q (afasroutines.f90:257-327, field 2): parent q(mb) =
// Restriction2D/3D (gridutilities.f90:103-126, :437-466) of the child's q,
// the sum left to right and then the product, as the FP64 path's kernel.
template <int NV, int DIM>
__device__ __forceinline__ void s_fill64(const PatchDev* __restrict__ P, double* pool, const Blk b, int tid, int push,
                                         const UniBC& bc, const ProbParams& pp) {
  const PatchDev& p = P[b.patch];
  int ci, cj, ck;
  if (!interior_cell<DIM>(p.cmx, b.start + tid, ci, cj, ck)) return;
  const PatchDev& par = P[p.parent];
  const int i = 2 * ci, j = 2 * cj, k = DIM == 3 ? 2 * ck : 0;
  double w[NV];
#pragma unroll
  for (int v = 0; v < NV; v++) {
    const double* q = pool + p.oq + v * p.sq;
    auto at = [&](int a, int b2, int c) { return q[gofs<DIM>(p.qn, a, b2, c)]; };
    double val;
    if (DIM == 2) {
      double s = __dadd_rn(__dadd_rn(__dadd_rn(at(i, j, 0), at(i - 1, j, 0)), at(i, j - 1, 0)), at(i - 1, j - 1, 0));
      val = __dmul_rn(0.25, s);
    } else {
      double s = at(i, j, k);
      s = __dadd_rn(s, at(i - 1, j, k));
      s = __dadd_rn(s, at(i, j - 1, k));
      s = __dadd_rn(s, at(i - 1, j - 1, k));
      s = __dadd_rn(s, at(i, j, k - 1));
      s = __dadd_rn(s, at(i - 1, j, k - 1));
      s = __dadd_rn(s, at(i, j - 1, k - 1));
      s = __dadd_rn(s, at(i - 1, j - 1, k - 1));
      val = __dmul_rn(0.125, s);
    }
    w[v] = val;
  }
  const int pi = p.mb[0] + ci - 1, pj = p.mb[1] + cj - 1, pk = DIM == 3 ? p.mb[2] + ck - 1 : 0;
  for (int v = 0; v < NV; v++) pool[par.oq + v * par.sq + gofs<DIM>(par.qn, pi, pj, pk)] = w[v];
  if (push) s_push<Push64<NV>, DIM>(pool + par.oq, par, pi, pj, DIM == 3 ? pk : 1, w, bc, pp);
}

// the FP64 residual partial sums of k_mx_norm, by one group of 256 threads
// (group g of its CTA) for padded block group b
template <class PL, int DIM>
__device__ __forceinline__ void s_norm(const PatchDev* __restrict__ P, double* pool, const Blk* __restrict__ blk,
                                       int b, int u, int g, const ProbParams& pp, double* partial,
                                       double (*red)[kBlock / 32]) {
  constexpr int NV = PL::kNV;
  double s[NV];
  bool any = false;
  for (int v = 0; v < NV; v++) s[v] = 0.0;
  for (int sub = 0; sub < kNormCells; sub++) {
    const Blk bb = blk[b * kNormCells + sub];
    if (bb.patch < 0) break;
    const PatchDev& p = P[bb.patch];
    int i, j, k;
    if (!interior_cell<DIM>(p.mx, bb.start + u, i, j, k)) continue;
    any = true;
    const double* q = pool + p.oq;
    long long sy = p.qn[0], sz = (long long)p.qn[0] * p.qn[1];
    long long c = gofs<DIM>(p.qn, i, j, k);
    long long fc = iofs<DIM>(p.mx, i, j, k);
    double r[NV];
    PL::template op<DIM>(q, c, sy, sz, p.sq, QoldView{pool + p.oqold + c, sy, sz, p.sq}, p.c, pp, r);
    for (int v = 0; v < NV; v++) {
      double e = pool[p.of + v * p.sf + fc] - r[v];
      pool[p.orf + v * p.sf + fc] = e;
      s[v] = fma(e, e, s[v]);
    }
  }
  warp_sums<NV>(s, red, u >> 5, u & 31, __any_sync(0xffffffffu, any));
  group_barrier(g);
  if (u < NV) {  // a thread a variable
    double t = 0.0;
    for (int m = 0; m < kBlock / 32; m++) t += red[u][m];
    partial[NV * b + u] = t;
  }
  group_barrier(g);
}

// The final sum of launch_norm_finish (one stage: nb <= 2048 partials) by
// the T threads of one CTA: the sums of its 1024 threads and their trees,
// bit for bit.  Sums of nothing are left out, as there: with 129 partials 5
// warps add instead of 32.  Thread 0 returns the variables' sums.
template <int NV, int T>
__device__ __forceinline__ void s_finish(const double* partial, int nb, double (*r2)[32], double* red0) {
  constexpr int kF = 1024;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int warps = min(32, (nb + 31) / 32);  // emulated warps that hold a partial
  for (int x = w; x < warps; x += T / 32) {
    double t[NV];
    const int n = x * 32 + lane;
    for (int v = 0; v < NV; v++) t[v] = n < nb ? partial[NV * n + v] : 0.0;
    if (x * 32 + kF < nb)
      for (int v = 0; v < NV; v++) t[v] += n + kF < nb ? partial[NV * (n + kF) + v] : 0.0;
    warp_sums<NV>(t, r2, x, lane, true);
  }
  __syncthreads();
  if (w == 0) {
    double t[NV];
    for (int v = 0; v < NV; v++) t[v] = lane < warps ? r2[v][lane] : 0.0;
    for (int o = 16; o > 0; o >>= 1)
      if (o < warps)
        for (int v = 0; v < NV; v++) t[v] += __shfl_down_sync(0xffffffffu, t[v], o);
    if (lane == 0)
      for (int v = 0; v < NV; v++) red0[v] = t[v];
  }
}

template <class PL, int DIM, int T>
struct SolveRun {
  const PatchDev* __restrict__ P;
  double* pool;
  float* fpool;
  double* partial;
  ProbParams pp;
  MxParams mp;
  const Blk* bpool;   // the image's block pool (shared memory)
  const int* spool;   // the image's stage pool
  const int* ppool;   // the image's part pool
  float* sdata;       // this CTA's FP32 data area (shared memory)
  int lg;             // log2 of the units per tile of the FP32 work lists
  UniBC ubc;
  const UniDim* dims;  // of the uniform levels (shared memory)
  const PackedGhost* sops;  // this CTA's FP32 ghost operations in shared memory, or null
  const PackedGhost* gops;  // the same in global memory, from this CTA's segment on
  int rank, ctas;

  __device__ __forceinline__ void sync(bool cluster) const {
    if (cluster) cluster_barrier();
    else __syncthreads();
  }

  // the blocks of a partitioned list this CTA works on (all of them in a solo block)
  template <typename F>
  __device__ __forceinline__ void owned(const SolvePhase& f, bool cluster, F&& unit) const {
    const Blk* blk = bpool + f.blk;
    const int* pt = ppool + f.part;
    const int lo = cluster ? pt[rank] : pt[0], hi = cluster ? pt[rank + 1] : pt[ctas];
    const int u = threadIdx.x & ((1 << lg) - 1);
    for (int b = lo + (int)(threadIdx.x >> lg); b < hi; b += T >> lg) unit(blk[b], u);
  }

  // one phase by the threads t0 = 0 .. nt-1 of the scope (the cluster, or
  // this CTA alone)
  __device__ __forceinline__ void exec(const SolvePhase& f, int t0, int nt, bool cluster,
                                       double (*red)[PL::kNV][kBlock / 32]) const {
    constexpr int nr = PL::kNV;
    // FP64 work is dealt a warp to each CTA in turn: its instructions take
    // their SM's FP64 unit 64 cycles each
    const int d0 = cluster ? (((int)threadIdx.x >> 5) * ctas + rank) * 32 + ((int)threadIdx.x & 31) : t0;
    switch (f.op) {
      case kTRelax:
        if (f.arg & kPushGhosts)
          owned(f, cluster, [&](const Blk& b, int u) { s_relax_push<PL, DIM>(P, fpool, b, u, f.arg, mp, ubc); });
        else
          owned(f, cluster, [&](const Blk& b, int u) { u_relax_any<PL, DIM, true>(P, fpool, b, u, f.arg, mp); });
        break;
      case kTRestrict:
        if (f.arg & kPushGhosts)
          owned(f, cluster, [&](const Blk& b, int u) { s_restrict_push<nr, DIM>(P, fpool, b, u, ubc); });
        else
          owned(f, cluster, [&](const Blk& b, int u) { u_restrict<DIM, true>(P, fpool, b, u, nr); });
        break;
      case kTRing:
        owned(f, cluster, [&](const Blk& b, int u) { u_coarse_ring<DIM, true>(P, fpool, b, u, nr, f.arg); });
        break;
      case kTLoad:
        owned(f, cluster, [&](const Blk& b, int u) { u_coarse_load<PL, DIM, true>(P, fpool, b, u, mp); });
        break;
      case kTProlong:
        owned(f, cluster, [&](const Blk& b, int u) { u_prolong<DIM, true>(P, fpool, b, u, nr); });
        break;
      case kSPrep:
        owned(f, cluster, [&](const Blk& b, int u) { u_prep<PL, DIM, true>(P, pool, fpool, b, u, f.arg, pp); });
        break;
      case kSUpdate:
        owned(f, cluster, [&](const Blk& b, int u) { u_update<DIM, true>(P, pool, fpool, b, u, nr, f.arg); });
        break;
      case kTGhost: {
        // stage s: this CTA's operations st[2*(s*ctas + r)] .. st[2*(s*ctas + r) + 1]
        // of its own list (inside a solo block CTA 0 holds every one)
        const int* st = spool + f.stage;
        for (int s = 0; s < f.nstages; s++) {
          const int lo = st[2 * (s * ctas + rank)], hi = st[2 * (s * ctas + rank) + 1];
          for (int t = lo + (int)threadIdx.x; t < hi; t += T) {
            const GhostOp g = ghost_op(sops ? sops[t] : gops[t]);
            ghost32_apply<true, nr>(P, fpool, g, nr);
          }
          if (s + 1 < f.nstages) sync(cluster);
        }
        break;
      }
      case kSGhost64: {
        const int* st = spool + f.stage;
        for (int s = 0; s < f.nstages; s++) {
          for (int t = st[s] + d0; t < st[s + 1]; t += nt) {
            const GhostOp g = f.ops[t];
            s_ghost64<PL::kNV>(P, pool, g, pp);
          }
          if (s + 1 < f.nstages) sync(cluster);
        }
        break;
      }
      case kSUniGhost: {
        const PatchDev& p = P[f.n];
        const int N = DIM == 3 ? p.mx[2] : p.mx[1];
        const uni::Geo g{p.mx[0], p.mx[1], N, 0, N, p.qn[0], p.qn[0] * p.qn[1], (int)p.sq};
        uni::set_ghost<Push32<nr>, DIM>(fbase<true>(fpool, p) + p.eq, g, dims[f.arg], t0, nt, ubc, 0);
        break;
      }
      case kSClear: {
        // the range of the FP32 pool, and this CTA's part of the e arrays
        // held in shared memory (offset, length) at part[2*rank]
        for (long long t = t0; t < f.len; t += nt) fpool[f.a + t] = 0.0f;
        if (f.part >= 0) {
          const int o = ppool[f.part + 2 * rank], n = ppool[f.part + 2 * rank + 1];
          for (int t = threadIdx.x; t < n; t += T) sdata[o + t] = 0.0f;
        }
        break;
      }
      case kSFill64: {
        const Blk* blk = bpool + f.blk;
        for (int b = d0 >> 5; b < f.n; b += nt >> 5)
          s_fill64<nr, DIM>(P, pool, blk[b], d0 & 31, f.arg & kPushGhosts, ubc, pp);
        break;
      }
      case kSNorm: {
        const Blk* blk = bpool + f.blk;
        const int g = threadIdx.x >> 8;
        for (int b = t0 >> 8; b < f.n; b += nt >> 8) s_norm<PL, DIM>(P, pool, blk, b, t0 & 255, g, pp, partial, red[g]);
        break;
      }
      default:
        break;
    }
  }
};

template <class PL, int DIM, int T>
__global__ void __launch_bounds__(T, 1)
    k_mx_solve(const unsigned char* __restrict__ img, SolveImage im, double* pool, float* fpool, SolveCtl* ctl,
               double* res, double* partial, ProbParams pp, MxParams mp) {
  constexpr int NV = PL::kNV;
  __shared__ double red[T / 256][NV][kBlock / 32];
  __shared__ double r2[NV][32];
  // every CTA stages the read-only program image after its data area and
  // its ghost operations: phases, patch table, block, stage and part pools
  unsigned char* const simg = solve_smem + im.data + im.ops;
  for (int x = threadIdx.x; x < im.bytes / 16; x += T)
    reinterpret_cast<int4*>(simg)[x] = reinterpret_cast<const int4*>(img)[x];
  __syncthreads();
  const int rank = (int)cluster_rank(), ctas = (int)cluster_ctas();
  const int* seg = reinterpret_cast<const int*>(simg + im.off_part) + im.seg;
  const PackedGhost* gops = ctl->ops + seg[rank];
  PackedGhost* sops = nullptr;
  if (im.ops_smem) {  // this CTA's FP32 ghost operations, as words
    sops = reinterpret_cast<PackedGhost*>(solve_smem + im.data);
    const int nw = (seg[rank + 1] - seg[rank]) * (int)(sizeof(PackedGhost) / 4);
    for (int x = threadIdx.x; x < nw; x += T) reinterpret_cast<int*>(sops)[x] = reinterpret_cast<const int*>(gops)[x];
  }
  // the data areas of the other CTAs are written from the first phase on:
  // every CTA of the cluster is running before any of them starts
  cluster_barrier();
  const SolvePhase* ph = reinterpret_cast<const SolvePhase*>(simg);
  const SolveRun<PL, DIM, T> R{reinterpret_cast<const PatchDev*>(simg + im.off_patches),
                               pool,
                               fpool,
                               partial,
                               pp,
                               mp,
                               reinterpret_cast<const Blk*>(simg + im.off_blk),
                               reinterpret_cast<const int*>(simg + im.off_stage),
                               reinterpret_cast<const int*>(simg + im.off_part),
                               reinterpret_cast<float*>(solve_smem),
                               im.tile_log2,
                               im.ubc,
                               reinterpret_cast<const UniDim*>(simg + im.off_dims),
                               sops,
                               gops,
                               rank,
                               ctas};
  const int nt = ctas * T, t0 = rank * T + (int)threadIdx.x;
  const int body = ctl->body, nph = ctl->nph, maxv = ctl->maxv, errortype = ctl->errortype;
  const double tol = ctl->tol, count = ctl->count;
  __shared__ int stop;  // set by thread 0 after each finish
  long long* trace = (rank == 0 && threadIdx.x == 0) ? ctl->trace : nullptr;
  if (trace) trace[nph] = clock64();
  for (int it = 0; it <= maxv; it++) {
    // it = 0: the prologue, phases [0, body); then the loop body once per V-cycle
    const int x0 = it == 0 ? 0 : body, x1 = it == 0 ? body : nph;
    for (int x = x0; x < x1; x++) {
      const SolvePhase f = ph[x];
      if (f.op == kSSolo) {
        if (rank == 0)
          for (int y = x + 1; y <= x + f.n; y++) {
            R.exec(ph[y], threadIdx.x, T, false, red);
            __syncthreads();
          }
        x += f.n;
        cluster_barrier();
        if (trace && it <= 1) trace[x] = clock64();
        continue;
      }
      if (f.op == kSFinish) {
        // every CTA sums the partials in the same order and takes the same
        // decision; CTA 0 records it
        double comp[NV];  // thread 0's
        s_finish<NV, T>(partial, f.n, r2, comp);
        if (threadIdx.x == 0) {
          double sum = comp[0];
          for (int v = 1; v < NV; v++) sum = sum + comp[v];
          double r;
          if (errortype == 1) {
            r = sqrt(sum / count);  // ErrorAFAS, afasroutines.f90:135
          } else {
            double cells = count / NV;
            r = sqrt(comp[0] / cells);
            for (int v = 1; v < NV; v++) {  // MAXVAL of the component errors, :146-153
              double e = sqrt(comp[v] / cells);
              r = e > r ? e : r;
            }
          }
          const bool nonfinite = !isfinite(r);
          const bool conv = !nonfinite && r < tol;
          stop = conv || nonfinite || it == maxv;
          if (rank == 0) {
            if (!nonfinite) res[it - 1] = r;
            ctl->norm[0] = r;
            ctl->norm[1] = sum;
            ctl->ncycles = it;
            ctl->converged = conv;
            ctl->nonfinite = nonfinite;
            ctl->stop = stop;
          }
        }
        __syncthreads();
      } else {
        R.exec(f, t0, nt, true, red);
      }
      if (f.bar) cluster_barrier();
      if (trace && it <= 1) trace[x] = clock64();
    }
    if (it > 0 && stop) break;
  }
}

}  // namespace mx
}  // namespace bsamg
