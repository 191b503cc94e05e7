// Launchers of the device kernels (one function per kernel family).  Every
// launcher enqueues on the given stream and returns the number of kernel
// launches it issued; the caller checks cudaGetLastError().
#pragma once
#include <cuda_runtime.h>

#include <utility>

#include "internal.h"

namespace bsamg {

constexpr int kNormOutLen = 8 + 3 * 128;

// A stream and how launch_after uses it: grids of up to `early` CTAs as
// programmatic dependents, larger ones in the plain order.
constexpr unsigned kEarlyCtas = 1024, kEarlyCtas64 = 152;
struct LaunchStream {
  cudaStream_t s = nullptr;
  unsigned early = kEarlyCtas;
  LaunchStream() = default;
  LaunchStream(cudaStream_t st) : s(st) {}
  operator cudaStream_t() const { return s; }
};

struct LaunchCtx {
  const PatchDev* P;  // device patch table
  double* pool;       // device FP64 pool
  float* fpool;       // device FP32 pool (mixed path), may be null
  LaunchStream s;
  ProbParams pp;
  int ndims;
};

// work-list kinds: what one unit of a level's block list is
enum Kind : int {
  kKindColor = 0,     // one slot of a colour row: ceil(mx1/2) * mx2 * mx3
  kKindInterior = 1,  // one interior cell: mx1*mx2*mx3
  kKindCoarse = 2,    // one coarse cell under a child: cmx1*cmx2*cmx3
  kKindCGhost = 3,    // one ghosted coarse cell: (cmx+2)^d
  kKindFGhost = 4,    // one ghosted fine cell: (mx+2)^d
  kKindProl = 5,      // one coarse index -gs..cmx+gs per dimension under a child: (cmx+1+2gs)^d
  kNKind = 6
};

// One phase of a V-cycle's coarse tail run inside one thread block (the
// operations the separate launches of those levels would run, recorded on
// the host).  kTRing: the coarse ring (arg 0) or CorrectFine's first step
// (arg 1); kTRelax: arg = ipass; kTFill: FillDownLevel, arg = field.
enum TailOp : int { kTRelax = 0, kTRestrict = 1, kTRing = 2, kTLoad = 3, kTProlong = 4, kTGhost = 5, kTFill = 6 };
// Flag of a relaxation's ipass on the correction's coarsest level: the
// smoother computes in FP64 (FP32 storage), the coarse solve of the
// V-cycle at the reference's precision.
constexpr int kRelax64 = 4;
// recorded for the one-launch solve: the operation writes the ghost images of
// the cells of a uniform level that it sets (restriction: of the parent's), and
// no ghost program follows
constexpr int kPushGhosts = 16;
struct TailPhase {
  int op, arg, nblk, nstages;
  const Blk* blk;
  const GhostOp* ops;
  const int* stage_off;
};

// Marks, while a solve program is recorded, the start of the coarse end of
// a V-cycle that one CTA runs alone (nblk = number of phases that follow).
constexpr int kTSolo = 7;

// The whole mixed-precision solve of a hierarchy with refinement levels as
// one program executed by a single thread-block cluster (kern_solve.cuh):
// the FP32 correction V-cycle's operations (ops 0-5, as TailOp), the FP64
// operations of the defect-correction loop around it, and the exit test.
enum SolveOp : int {
  kSClear = 8,     // fpool[a .. a+len) = 0
  kSPrep = 9,      // base planes and g of a level (arg = mode of mx_prep)
  kSUpdate = 10,   // qbar += e over the ghosted cells, e = 0, base refresh (arg = variables refreshed)
  kSFill64 = 11,   // FillDown of q in FP64 (FillDownLevel, field 2)
  kSGhost64 = 12,  // an FP64 ghost program
  kSNorm = 13,     // FP64 residual of the finest level: rf and n partial sums (padded interior list)
  kSFinish = 14,   // one CTA: the deterministic final sum, the residual record and the exit decision
  kSUniGhost = 16, // the ghosts of the correction on a uniform level (arg = -level, n = its patch)
  kSSolo = 15      // the next n phases run in CTA 0 alone (barriers of that CTA between them)
};
// FP32 operations (0-5, kSClear, kSPrep, kSUpdate) take their work by
// owner: each CTA the blocks (ghost operations) of the patches it owns,
// part[rank] .. part[rank+1] of the phase's list (of each stage), CTA 0
// all of them inside a solo block.  FP64 operations spread their list over
// all threads of the cluster.
struct SolvePhase {
  int op, arg, n, nstages;
  int bar;    // a cluster barrier follows the phase
  int blk;    // the phase's work list: first entry in the program image's block pool
  int stage;  // ghost programs: first entry of their stage offsets in the image's stage pool
              // (FP64: nstages+1 offsets; FP32: for stage s and CTA r, the pair at 2*(s*ctas + r))
  int part;   // owner partition: first of ctas+1 entries in the image's part pool (-1: none)
  const GhostOp* ops;  // a ghost program's operations (global memory)
  long long a, len;    // kSClear: the range of the FP32 pool
};
// Uniform levels (kern_uni.cuh).  UniBC: per dimension 0 periodic, 1
// physical faces (UserBC with the plugin's mask).
struct UniBC {
  int phys[3];
  int mask;
};
// The program image every CTA of a solve copies into its shared memory at
// the start, after a data area of `data` bytes that holds the FP32 arrays
// of the patches it owns in distributed shared memory: the phases at
// offset 0, then the patch table, the block, stage and part pools (byte
// offsets from the image's start, 16-byte aligned).  Read-only data read
// from shared memory is not lost at a cluster barrier, whose acquire
// discards what the L1 cache holds.
struct SolveImage {
  int bytes, data, off_patches, off_blk, off_stage, off_part;
  int off_dims;   // the UniDim of level -l at index l (uniform levels)
  // the FP32 ghost operations are ordered by CTA: CTA r's are [seg[r],
  // seg[r+1]) of the program's operation array (seg: ctas+1 entries of the
  // part pool at off_seg); when ops_smem, each CTA stages its own after its
  // data area (ops bytes reserved per CTA)
  int seg, ops_smem, ops;
  UniBC ubc;      // boundary conditions of the uniform levels (kPushGhosts)
  int tile_log2;  // FP32 work lists are split into tiles of 2^tile_log2 units (at most 256)
};
constexpr int kSolveSmemMax = 222 * 1024;  // shared memory of a CTA: data area, image, ghost operations
// An FP32 ghost operation of a solve in seven words (GhostOp takes eleven):
// an adaptive level's operations then fit beside the data area and the image,
// where each cost a trip to the L2 cache in every ghost stage.  The cells an
// interpolation reads lie within two rows (planes) of the first; the patches
// are 16-bit indices (solve_build checks both).
struct PackedGhost {
  unsigned type_mask;  // type | mask << 3
  unsigned short dp, sp;
  int dcell, s0, c0;
  short s1, c1, c2, c3;  // relative to s0 and c0
};
__host__ __device__ inline PackedGhost solve_op(const GhostOp& g) {
  PackedGhost o;
  o.type_mask = (unsigned)g.type | (unsigned)g.mask << 3;
  o.dp = (unsigned short)g.dp, o.sp = (unsigned short)g.sp;
  o.dcell = g.dcell, o.s0 = g.s0, o.c0 = g.c0;
  o.s1 = (short)(g.s1 - g.s0);
  o.c1 = (short)(g.c1 - g.c0), o.c2 = (short)(g.c2 - g.c0), o.c3 = (short)(g.c3 - g.c0);
  return o;
}
__host__ __device__ inline GhostOp ghost_op(const PackedGhost& o) {
  GhostOp g;
  g.type = (int)(o.type_mask & 7u), g.mask = (int)(o.type_mask >> 3);
  g.dp = o.dp, g.sp = o.sp;
  g.dcell = o.dcell, g.s0 = o.s0, g.s1 = o.s0 + o.s1;
  g.c0 = o.c0, g.c1 = o.c0 + o.c1, g.c2 = o.c0 + o.c2, g.c3 = o.c0 + o.c3;
  return g;
}
// Control block of a solve launch (device memory); the residual of V-cycle
// it (1-based) follows it at res[it-1].
struct SolveCtl {
  int body, nph;      // first phase of the loop body, phases in the program
  int maxv, errortype;
  double tol, count;  // exit tolerance, ErrorAFAS denominator of the finest level
  int nb, nrvars;     // partial sums of the norm, variables
  // results
  int ncycles, converged, nonfinite, stop;
  double norm[2];     // the last norm and its raw sum
  const PackedGhost* ops;  // the program's FP32 ghost operations, CTA after CTA
  // when set: CTA 0's clock at the end of every phase of the prologue and
  // the first outer iteration (trace[x], cycles of the SM it runs on), and
  // at the start (trace[nph])
  long long* trace;
};
// launch shape of the solve kernel: CTAs in the cluster, threads per CTA
struct SolveShape {
  int ctas, threads;
  int tile;  // units per tile of the FP32 work lists (32, 64, 128 or 256)
};

// Division by d as a multiplication by m = ceil(2^32 / d) (0: d = 1)
struct UniDiv {
  int d;
  unsigned m;
};
// the divisors of a level's index decoding: (n0+1)/2, n0, n1, the ghosted
// extents, the coarse image's interior, +1 and ghosted extents, and the cells
// of a plane's frame (3D) of the level and of its coarse image
struct UniDim {
  UniDiv hx, n0, n1, e0, e1, c0, c1, cp0, cp1, ce0, ce1, ring, cring;
};
inline UniDim uni_dim(const int* n) {
  auto dv = [](int d) { return UniDiv{d, d <= 1 ? 0u : 0xFFFFFFFFu / (unsigned)d + 1u}; };
  const int c0 = n[0] / 2, c1 = n[1] / 2;
  return UniDim{dv((n[0] + 1) / 2), dv(n[0]), dv(n[1]), dv(n[0] + 2), dv(n[1] + 2), dv(c0 > 0 ? c0 : 1), dv(c1 > 0 ? c1 : 1),
                dv(c0 + 1), dv(c1 + 1), dv(c0 + 2), dv(c1 + 2), dv(2 * (n[0] + 2) + 2 * n[1]),
                dv(2 * (c0 + 2) + 2 * c1)};
}
// a level's table entry and divisors, as a kernel argument
struct UniPatch {
  PatchDev p;
  UniDim d;
};
inline UniPatch uni_patch_of(const PatchDev& p) { return UniPatch{p, uni_dim(p.mx)}; }
// One level of a cluster's V-cycle: its patch, extents, the most rows of the
// slowest dimension a CTA holds, the rows per row of the partition (0: CTA 0
// holds the level alone) and where its arrays start in every CTA's shared
// memory (elements): q, f, the coarse image, and the frozen data (qold or
// base planes).
struct UniLev {
  int patch;
  int n[3];
  int maxr, mul;
  int q, f, c, x;
  UniDim d;
};
// the partition's rows of one CTA
struct UniRank {
  short row0, rows;
};
struct UniCycle {
  UniLev L[kNLev];  // finest first
  UniRank R[16];
  int nl, ctas, threads, nsmooth;
  int scratch;      // start of a CTA's residual scratch (elements)
  UniBC bc;
};
constexpr int kUniThreads = 512;           // most threads of a CTA
constexpr int kUniFillThreads = 1024;
constexpr int kUniSmemMax = 200 * 1024;    // dynamic shared memory of a CTA

// A contiguous run of pool elements staged in shared memory by a tail
// kernel: pool[g .. g+n) <-> smem[s .. s+n); written back when out != 0.
struct StageSeg {
  long long g;
  int s, n, out, pad;
};
constexpr int kTailSmemMax = 160 * 1024;  // shared-memory budget of a staged tail

// ---- plain FP64 path (fp64.cu, built with --fmad=false) ----
int launch_relax(const LaunchCtx& c, const Blk* blk, int nblk, int ipass);
int launch_restrict_q(const LaunchCtx& c, const Blk* blk, int nblk);
int launch_coarse_ghost(const LaunchCtx& c, const Blk* blk, int nblk);
int launch_coarse_load(const LaunchCtx& c, const Blk* blk, int nblk);
int launch_correct_a(const LaunchCtx& c, const Blk* blk, int nblk);
// qc of every patch in blk = its parent's q under it, ghost rings included
int launch_qc_from_parent(const LaunchCtx& c, const Blk* blk, int nblk);
int launch_correct_b(const LaunchCtx& c, const Blk* blk, int nblk);
int launch_fill_down(const LaunchCtx& c, const Blk* blk, int nblk, int field);
int launch_get_source(const LaunchCtx& c, const Blk* blk, int nblk);
int launch_update_source(const LaunchCtx& c, const Blk* blk, int nblk);
// partial sums of rf^2 (nrvars per CTA) -> partial[norm_partials(nblk)*nrvars]:
// one CTA per norm_group(nblk) consecutive blocks of the work list, as many
// CTAs as are resident at once (four an SM), so that the last wave is a full
// one and the FP64 shuffle reduction (10 additions a thread for two
// variables, beside about 14 FP64 instructions a cell) is paid once a group;
// a small level takes one block a CTA to reach every SM (a 128^2 level in 16
// CTAs of four blocks: 17 us, in 64: 6 us).
constexpr int kNormPartialsMax = 608;
inline int norm_group(int nblk) { return nblk <= kNormPartialsMax ? 1 : (nblk + kNormPartialsMax - 1) / kNormPartialsMax; }
inline int norm_partials(int nblk) { return (nblk + norm_group(nblk) - 1) / norm_group(nblk); }
int launch_norm_partial(const LaunchCtx& c, const Blk* blk, int nblk,
                        double* partial, int store_rf);
// deterministic final sum; writes out[0] = norm, out[1] = raw sum,
// and nonfinite[0] = 0 when the norm is finite, 1 otherwise (nothing when
// nonfinite is null).  With `host` (pinned memory) the record a host reads
// goes there too: host[0] and host[1] as out, the flag as an int at host + 8;
// with `one` the norm also goes to *one.  out must hold
// kNormOutLen doubles (out[8 ..] is scratch of the two-stage sum); the
// partials hold nrvars values per block.
int launch_norm_finish(LaunchStream s, const double* partial, int nblk,
                       int nrvars, double count, int errortype, double* out,
                       int* nonfinite, double* host = nullptr, double* one = nullptr);
int launch_ghost_stage(const LaunchCtx& c, const GhostOp* ops, int n);

// ---- after-step statistics and uniform-mesh output (io.cu, --fmad=false) ----
// partial[2*(pofs + b)] = (mass, energy) of block b of a level's interior
// list (coarse = false) or, negated, of the parent cells of its coarse list
int launch_stats(const LaunchCtx& c, const Blk* blk, int nblk, bool coarse, int mass, int energy, double* partial,
                 int pofs);
int launch_stats_finish(cudaStream_t s, const double* partial, int n, double* out);
// F = mass-corrected prolongation of the uniform (n+2)^d block A (one variable)
int launch_uniform_prolong(cudaStream_t s, int ndims, const double* A, double* F, const int n[3]);
// the seeded spinodal start of one CH patch (q: its ghosted q, two planes of sq)
int launch_seed_spinodal(cudaStream_t s, int ndims, int mbc, double* q, long long sq, const int mx[3], unsigned long long seed,
                         double mean, double amp, double eps2, double h);
// a patch's q(0:mx+1) (nv variables; oq the offset of its cell (0,0,0))
// into the uniform block U (extents un)
int launch_uniform_scatter(cudaStream_t s, int ndims, const double* pool, long long oq, long long sq, const int qn[3],
                           const int mx[3], const int g[3], double* U, const int un[3], int nv);
// A ghost program of several stages and few operations runs in one CTA, its
// stages apart by CTA barriers; otherwise a launch a stage.  One CTA takes a
// round of 256 operations (FP64: some 20 dependent instructions of 64 cycles)
// after the other: a program of one stage and 1000 operations 14 us, its stage
// over the GPU 6.5.
inline bool ghost_in_one_cta(int nstages, int nops) { return nstages > 1 && nops <= 512; }
int launch_ghost_program_1cta(const LaunchCtx& c, const GhostOp* ops,
                              const int* stage_off, int nstages);
// the recorded coarse tail of an FP64 V-cycle, one block
int launch_tail(const LaunchCtx& c, const TailPhase* ph, int nph);
// the same on arrays staged in shared memory (shadow: the patch table that
// addresses them); tail_smem_attributes raises the dynamic shared-memory
// limit of a plugin's kernels to kTailSmemMax (0 on success)
int launch_tail_smem(const LaunchCtx& c, const PatchDev* shadow, const TailPhase* ph, int nph, const StageSeg* segs,
                     int nsegs, int smem_bytes);
int tail_smem_attributes(int problem);

#ifdef __CUDACC__
// Programmatic dependent launch: a kernel launched by launch_after may be set
// up, its CTAs resident, while the kernel before it in the stream still runs,
// which takes part of the launch latency off chains of small kernels (a V-cycle
// of 30 to 110 launches: 2 to 5 % of it).  Its first statement is
// after_previous(): it lets the next kernel do the same and waits until the
// one before has finished and its writes are visible.  CTAs that wait hold
// slots, which is why not every launch is made so (Hier::launch_order):
// - Grids of many waves: their early CTAs wait in the slots of the running
//   kernel's last wave (a mixed step at 256^3 5.43 -> 5.56 ms).
// - FP64 solves, whose kernels are bound by the FP64 unit and the integer
//   pipe, want their CTAs spread evenly over the SMs, and early ones go where
//   the running kernel left room.  In 2D, grids of up to a CTA an SM gain (a
//   step of five V-cycles, early | plain: 128^2 0.882 | 0.909 ms, 256^2 1.146 |
//   1.181; with grids of up to 1024 CTAs 512^2 lost, 1.964 | 1.763); in 3D all
//   lost (64^3 1.976 | 1.770, 128^3 4.953 | 4.738; up to a CTA an SM still
//   2 to 4 %; adaptive growth 33.6 | 31.4).
// - Hierarchies that share the GPU with others: their CTAs hold the others'
//   slots (serving 200 requests a second, early launches 1820 steps/s and a
//   median of 310 ms, the plain order 2280 and 40 ms; see SolveRuns in hier.cu).
__device__ __forceinline__ void after_previous() {
  asm volatile("griddepcontrol.launch_dependents;\n\tgriddepcontrol.wait;" ::: "memory");
}
template <typename... P, typename... A>
inline void launch_after(void (*k)(P...), dim3 grid, dim3 block, size_t smem, LaunchStream s, A&&... a) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = (unsigned long long)grid.x * grid.y * grid.z <= s.early ? 1 : 0;
  cudaLaunchKernelEx(&cfg, k, std::forward<A>(a)...);
}
// the same for one cluster of `ctas` CTAs, the largest waiters there are: up to
// 16 SMs' shared memory
template <typename... P, typename... A>
inline cudaError_t launch_cluster(void (*k)(P...), int ctas, int threads, int smem, LaunchStream s, A&&... a) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = ctas;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = s.early ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, k, std::forward<A>(a)...);
}
#endif

}  // namespace bsamg
