// Convergence norm of one CH patch on caller-owned device buffers, with no
// allocation of any kind.
//
// Some callers cannot let a library call cudaMalloc: a host whose device
// memory is owned by its own allocator (a PyTorch caching allocator, a
// Fortran code with a fixed device-memory plan), or a serving loop that must
// not trigger the device-wide synchronisation cudaMalloc/cudaFree imply while
// other streams are busy.  This entry point computes ErrorAFAS
// (afasroutines.f90:113-233) of one CH patch from q and f the caller already
// has on the device and writes the norm to a device double the caller owns.
// Its only scratch -- one partial sum per block plus the final reduction's
// stage sums -- lives in a file-scope __device__ array of fixed size, so a
// patch may have at most BSAMG_NOALLOC_MAX_CELLS interior cells (256^3).
//
// The array exists once per device for the life of the process and every
// call on that device shares it: two calls whose kernels overlap on the GPU
// (different streams, no ordering between them) race on it.  Each call
// writes every partial it later reads, so nothing needs clearing between
// calls.  The first call on a device looks the array's device address up
// (cudaGetSymbolAddress, with that device current) and keeps it for the
// rest of the process; make that first call before any stream capture that
// includes this entry point.  The kept address does not survive
// cudaDeviceReset (the module is loaded again, possibly elsewhere): a host
// that resets a device must not call this entry point on it afterwards.
//
// Same arithmetic, block decomposition and final reduction as the
// hierarchy's norm (the partial kernel below is k_uni_norm's for one CH
// patch, built with --fmad=false like it, and the final sum is
// launch_norm_finish itself), so the two agree bit for bit.
#include <cuda_runtime.h>

#include <cstdint>
#include <mutex>

#include "../../include/bsamg.h"
#include "hier.h"
#include "internal.h"
#include "kern_fp64.cuh"
#include "launch.h"

namespace {

using namespace bsamg;

constexpr int kMaxBlocks = kNormPartialsMax;

// [0, 2*kMaxBlocks): per-CTA partial sums of rf^2 (two variables);
// [2*kMaxBlocks, 2*kMaxBlocks + kNormOutLen): the final reduction's output
// and stage sums (launch_norm_finish's `out`)
__device__ __align__(256) double g_norm_scratch[2 * kMaxBlocks + kNormOutLen];

std::mutex g_mu;
constexpr int kMaxDevices = 256;
double* g_scratch_ptr[kMaxDevices] = {};

int scratch_on_device(int dev, double** out) {
  if (dev < 0 || dev >= kMaxDevices) return BSAMG_ERR_UNSUPPORTED;
  std::lock_guard<std::mutex> lk(g_mu);
  if (!g_scratch_ptr[dev]) {
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_norm_scratch);
    if (e != cudaSuccess) return cuda_fail(e, "cudaGetSymbolAddress(g_norm_scratch)");
    g_scratch_ptr[dev] = static_cast<double*>(p);
  }
  *out = g_scratch_ptr[dev];
  return BSAMG_OK;
}

// Whether the final kernel stores the norm itself: to a double's address in
// memory of its own device.  Any other (unaligned, a peer's memory without
// access enabled) would fault there and is left to a copy.  Where there is one
// device its place is not asked for: a call on a small patch is bound by the
// host (11.7 us a call without, 13.2 with the question).
bool kernel_can_store(const double* p, int dev) {
  if (reinterpret_cast<uintptr_t>(p) % alignof(double)) return false;
  static const int devices = [] {
    int n = 0;
    return cudaGetDeviceCount(&n) == cudaSuccess ? n : 2;
  }();
  if (devices == 1) return true;
  cudaPointerAttributes at = {};
  if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
    cudaGetLastError();  // the copy reports it
    return false;
  }
  return at.type == cudaMemoryTypeManaged || (at.type == cudaMemoryTypeDevice && at.device == dev);
}

template <int DIM>
__device__ __forceinline__ double lap(const double* a, int c, int sy, int sz) {
  if (DIM == 2) return a[c + 1] + a[c - 1] + a[c + sy] + a[c - sy] - 4.0 * a[c];
  return fxp::lap6({a[c + 1], a[c - 1], a[c + sy], a[c - sy], a[c + sz], a[c - sz]}, a[c]);
}

// rf = f - Operator(q) (CH/problem.f90:393-422, :638-669) per interior cell,
// sums of rf^2 over `group` consecutive runs of kBlock cells per CTA, in the
// order of the hierarchy's norm on a one-patch level (whose blocks are the
// same runs of cells).  Bound by the FP64 unit and the integer ALU alike: 15
// FP64 instructions a cell, the Laplacians' sums on the integer pipe beside
// them (31 with all of them on the FP64 unit: 119 us for 160 x 96 x 128, now
// 79 with the final sum).
template <int DIM>
__global__ void __launch_bounds__(kBlock, 4) k_norm_single(const double* __restrict__ q, const double* __restrict__ f,
                                                        int mx0, int mx1, int mx2, const __grid_constant__ UniDim d,
                                                        int group, double c0, double c1,
                                                        double* __restrict__ partial) {
  __shared__ double red[2][kBlock / 32];
  double s[2] = {0.0, 0.0};
  const int cells = mx0 * mx1 * (DIM == 2 ? 1 : mx2);
  const int n0 = mx0 + 2, n1 = mx1 + 2, sy = n0, sz = n0 * n1;
  const int sq = DIM == 2 ? sz : sz * (mx2 + 2);
  for (int sub = 0; sub < group; sub++) {
    const int fc = (blockIdx.x * group + sub) * kBlock + (int)threadIdx.x;
    if (fc >= cells) break;
    int i, j, k;
    uni::inner_unit<DIM>(d.n0, d.n1, fc, i, j, k);
    const int c = DIM == 2 ? j * n0 + i : (k * n1 + j) * n0 + i;
    const double* a0 = q;
    const double* a1 = q + sq;
    double r0 = a0[c] - c0 * lap<DIM>(a1, c, sy, sz);
    double r1 = a1[c] - a0[c] * a0[c] * a0[c] + c1 * lap<DIM>(a0, c, sy, sz);
    double e0 = f[fc] - r0;
    double e1 = f[cells + fc] - r1;
    s[0] = fma(e0, e0, s[0]);
    s[1] = fma(e1, e1, s[1]);
  }
  block_sum<2>(s, red, partial);
}

}  // namespace

extern "C" int bsamg_ch_residual_norm_noalloc(const double* q, const double* f, int ndims, const int mx[3],
                                              double h, double dt, double eps, int errortype, double* norm_out,
                                              void* stream) {
  if (!q || !f || !mx || !norm_out || (ndims != 2 && ndims != 3) || (errortype != 1 && errortype != 2) ||
      !(h > 0.0))
    return BSAMG_ERR_ARG;
  long long cells = 1;
  for (int d = 0; d < ndims; d++) {
    if (mx[d] < 1) return BSAMG_ERR_ARG;
    cells *= mx[d];
  }
  if (cells > BSAMG_NOALLOC_MAX_CELLS) {
    cuda_fail(cudaSuccess, "bsamg_ch_residual_norm_noalloc: patch larger than BSAMG_NOALLOC_MAX_CELLS");
    return BSAMG_ERR_ARG;
  }
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return cuda_fail(e, "cudaGetDevice");
  double* scratch = nullptr;
  int rc = scratch_on_device(dev, &scratch);
  if (rc != BSAMG_OK) return rc;
  const bool store = kernel_can_store(norm_out, dev);
  // plugin coefficients exactly as the hierarchy computes them
  double h2 = h * h;
  double eps2 = eps * eps;
  double c0 = dt / h2, c1 = eps2 / h2;
  const int runs = (int)((cells + kBlock - 1) / kBlock), nblk = norm_partials(runs), group = norm_group(runs);
  const int n[3] = {mx[0], mx[1], ndims == 2 ? 1 : mx[2]};
  const UniDim d = uni_dim(n);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (ndims == 2)
    k_norm_single<2><<<nblk, kBlock, 0, s>>>(q, f, n[0], n[1], 1, d, group, c0, c1, scratch);
  else
    k_norm_single<3><<<nblk, kBlock, 0, s>>>(q, f, n[0], n[1], n[2], d, group, c0, c1, scratch);
  // the hierarchy's own final reduction (two stages above 2048 blocks);
  // no non-finite flag: a NaN or Inf input shows as a NaN or Inf norm
  double* out = scratch + 2 * kMaxBlocks;
  launch_norm_finish(s, scratch, nblk, 2, 2.0 * (double)cells, errortype, out, nullptr, nullptr,
                     store ? norm_out : nullptr);
  e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "bsamg_ch_residual_norm_noalloc launch");
  if (store) return BSAMG_OK;
  e = cudaMemcpyAsync(norm_out, out, sizeof(double), cudaMemcpyDeviceToDevice, s);
  return e == cudaSuccess ? BSAMG_OK : cuda_fail(e, "bsamg_ch_residual_norm_noalloc copy");
}
