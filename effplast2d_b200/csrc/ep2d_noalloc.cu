// ep2d_noalloc.cu -- the RVE averaging for callers that cannot allocate device memory.
//
// Some callers hold every byte of device memory through their own allocator (a host
// framework's caching allocator, a fixed pool sized at start-up) and may not call
// cudaMalloc: a library allocation would grow or fragment memory they account for,
// and cudaMalloc/cudaFree synchronise the device.  ep2d_average_fields_noalloc serves
// them: the caller passes its own device arrays and its own output buffer, and the
// reduction's per-block partial sums go to a fixed array in this file instead of to
// memory the library would allocate.
//
// The array is a file-scope __device__ variable: every GPU that loads the library holds
// it (kMaxBlocks x kSums doubles and the counts, 193 KiB) until the process exits.  Host code must not
// use its name as an address -- on the host the name is only a stand-in -- so the first
// call on each device looks its device address up with cudaGetSymbolAddress while that
// device is current, and passes that pointer to the kernels.  The address belongs to the
// device's current context: after a cudaDeviceReset the module is loaded again, possibly
// elsewhere, so the lookup is keyed on the context too and the first call in a new
// context repeats it.  That first call (per device, and again after a reset) should come
// before any stream capture.  Every call overwrites all the partials it later reads and
// leaves its count at zero, so nothing needs clearing between calls; calls that overlap on the GPU would share the
// array and race.
#include <cuda.h>

#include <atomic>
#include <cmath>
#include <mutex>
#include <string>

#include "ep2d.h"
#include "ep2d_rve.hpp"
#include "ep2d_types.hpp"

namespace ep2d {
namespace {

constexpr int kMaxBlocks = 2048;
constexpr int kMaxRowsPerBlock = 4;  // rows (ny - 2) up to 8192, i.e. ny <= 8194
constexpr int kMaxDevices = 64;
constexpr int kSums = 12;    // partial sums of a block: sigma 0-2, sigma_per 4-7, and the strains' sums below
constexpr int kThreads = 256;

// the partial sums, kMaxBlocks x kSums, and counts of blocks that have written theirs (zero
// between calls).  Calls take the counts in turn and each also clears the one half a turn away, so
// that calls which overlapped on the GPU against the contract leave nothing behind.
constexpr unsigned kTurns = 256;
struct AvgScratch {
  double part[kMaxBlocks * kSums];
  unsigned arrived[kTurns];
};
static __device__ __align__(256) AvgScratch g_avg_scratch;

std::mutex g_scratch_mu;
AvgScratch* g_scratch_dev[kMaxDevices] = {};
CUcontext g_scratch_ctx[kMaxDevices] = {};  // the context each cached address belongs to

// cuCtxGetCurrent through the runtime's driver entry point (no link against libcuda)
using CtxGetCurrentFn = CUresult (*)(CUcontext*);
CtxGetCurrentFn ctx_get_current() {
  static CtxGetCurrentFn fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q{};
    if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &p, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      p = nullptr;
    return reinterpret_cast<CtxGetCurrentFn>(p);
  }();
  return fn;
}

// The scratch array's device address on the current device, looked up once per device
// and context.
int scratch_on_current_device(AvgScratch** out) {
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= kMaxDevices)
    return fail(EP2D_ERR_NODEV, std::string("no current CUDA device: ") + cudaGetErrorString(e));
  CtxGetCurrentFn get = ctx_get_current();
  if (!get) return fail(EP2D_ERR_CUDA, "cuCtxGetCurrent is not available from the CUDA driver");
  // the context current on this thread; null before the runtime has made one current,
  // which the lookup below does (cudaGetSymbolAddress initialises the device's primary
  // context; nothing here allocates)
  CUcontext ctx = nullptr;
  if (get(&ctx) != CUDA_SUCCESS) ctx = nullptr;
  std::lock_guard<std::mutex> lk(g_scratch_mu);
  if (!ctx || !g_scratch_dev[dev] || g_scratch_ctx[dev] != ctx) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_avg_scratch);
    if (e != cudaSuccess || !p)
      return fail(EP2D_ERR_CUDA, std::string("cudaGetSymbolAddress of the averaging scratch: ") +
                                     cudaGetErrorString(e));
    if (!ctx && (get(&ctx) != CUDA_SUCCESS || !ctx))
      return fail(EP2D_ERR_CUDA, "no current CUDA context after the scratch lookup");
    g_scratch_dev[dev] = static_cast<AvgScratch*>(p);
    g_scratch_ctx[dev] = ctx;
  }
  *out = g_scratch_dev[dev];
  return EP2D_OK;
}

// Sums v[0..15] over the warp: each exchange halves the values a lane carries, 16 shuffles of
// a double instead of 5 for each of the 16 sums.  Lane l returns the sum of column warp_column(l).
__device__ __forceinline__ double warp_sums(double (&v)[16], int lane) {
#pragma unroll
  for (int n = 8; n >= 1; n >>= 1) {
    const bool up = lane & (2 * n);
#pragma unroll
    for (int k = 0; k < n; k++)
      v[k] = (up ? v[k + n] : v[k]) + __shfl_xor_sync(0xffffffffu, up ? v[k] : v[k + n], 2 * n);
  }
  return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
}
__device__ __forceinline__ int warp_column(int lane) { return lane >> 1; }

// The sums of EffPlast2D.cu:456-490 over the reference's own layout (P, tauXX, tauYY: nX
// per row; tauXY: nX - 1; Ux: nX + 1; Uy: nX) and the averages of :491-503, in one launch:
// every block writes the partial sums of its rows, and the last one to arrive adds them
// all, in block order per lane and then over lanes, so the result does not depend on
// which block that is.  The strains are summed as displacement differences and divided
// by dX and dY once, at the end, where each term was divided before: fewer roundings and no
// division in the loop.
//
// Bound by latency at the sizes in use (512^2: 12.6 MB, 1.9 us at the measured HBM rate): one
// or two rows per block, so that every SM has several blocks' loads in flight, few
// shuffles, and no second launch, whose one warp added the partials in a serial chain.  A call, back to
// back, before and now: 512^2 16.4 / 10.3 us (9.8 is what the caller's side of a call takes),
// 1024^2 28.7 / 14.4, 2048^2 72 / 44 (4.6 TB/s).
__global__ void __launch_bounds__(kThreads)
    k_average_reference_layout(long nX, long nY, double dX, double dY, const double* __restrict__ P,
                               const double* __restrict__ txx, const double* __restrict__ tyy,
                               const double* __restrict__ txy, const double* __restrict__ Ux,
                               const double* __restrict__ Uy, double nu0, int perOffsetX, int perOffsetY,
                               int rows_per_block, double div_all, double div_xy, double div_inner,
                               AvgScratch* __restrict__ scratch, unsigned turn, double* __restrict__ out) {
  double acc[16];
#pragma unroll
  for (int k = 0; k < 16; k++) acc[k] = 0.0;
  const long jb = 1 + (long)blockIdx.x * rows_per_block;
  const long je = (jb + rows_per_block < nY - 1) ? jb + rows_per_block : nY - 1;
  for (long j = jb; j < je; j++) {
    const bool inner_row = j > perOffsetY && j < nY - perOffsetY;
    for (long i = 1 + threadIdx.x; i < nX - 1; i += kThreads) {
      const long q = j * nX + i, c = j * (nX - 1) + i;
      const double pv = P[q], xv = txx[q], yv = tyy[q], cv = txy[c];
      const double zz = nu0 * (xv + yv - 2.0 * pv);
      acc[0] += xv - pv;
      acc[1] += yv - pv;
      acc[2] += cv + zz;
      if (inner_row && i > perOffsetX && i < nX - perOffsetX) {
        const long cm = c - (nX - 1);
        const long x0 = j * (nX + 1) + i, xm = x0 - (nX + 1), xp = x0 + (nX + 1);
        const long yp = q + nX;
        const double ux00 = Ux[x0], ux10 = Ux[x0 + 1], uy00 = Uy[q], uy01 = Uy[yp];
        acc[4] += xv - pv;
        acc[5] += yv - pv;
        acc[6] += 0.25 * (txy[cm - 1] + txy[cm] + txy[c - 1] + cv);
        acc[7] += zz;
        acc[8] += ux10 - ux00;
        acc[9] += uy01 - uy00;
        acc[10] += (ux00 - Ux[xm]) + (ux10 - Ux[xm + 1]) + (Ux[xp] - ux00) + (Ux[xp + 1] - ux10);
        acc[11] += (uy00 - Uy[q - 1]) + (Uy[q + 1] - uy00) + (uy01 - Uy[yp - 1]) + (Uy[yp + 1] - uy01);
      }
    }
  }
  __shared__ double red[16][kThreads / 32];
  __shared__ bool last;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const double sum = warp_sums(acc, lane);
  if (!(lane & 1)) red[warp_column(lane)][w] = sum;
  __syncthreads();
  if (threadIdx.x < kSums) {
    double v = 0.0;
    for (int q = 0; q < kThreads / 32; q++) v += red[threadIdx.x][q];
    scratch->part[(size_t)blockIdx.x * kSums + threadIdx.x] = v;
    __threadfence();  // before the block's arrival is counted
  }
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(&scratch->arrived[turn], 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();  // the other blocks' sums are read after the count
  // thread t adds column t % 16 of the blocks t / 16, t / 16 + 16, ...
  const int col = threadIdx.x & 15, first = threadIdx.x >> 4;
  double v = 0.0;
  if (col < kSums) {
#pragma unroll 8
    for (int b = first; b < (int)gridDim.x; b += kThreads / 16) v += __ldcg(&scratch->part[(size_t)b * kSums + col]);
  }
  v += __shfl_xor_sync(0xffffffffu, v, 16);
  __syncthreads();
  if (lane < 16) red[lane][w] = v;
  __syncthreads();
  if (threadIdx.x < kSums) {
    double t = 0.0;
    for (int q = 0; q < kThreads / 32; q++) t += red[threadIdx.x][q];
    red[threadIdx.x][0] = t;
  }
  __syncthreads();
  if (threadIdx.x == 0) scratch->arrived[turn] = scratch->arrived[(turn + kTurns / 2) % kTurns] = 0;
  if (threadIdx.x < NAVG) {
    // out: sigma[0..3], sigma_per[0..3], eps_per[0..2]; sigma[3] is never accumulated
    const int k = threadIdx.x;
    v = k == 3 ? 0.0 : red[k][0];
    if (k == 8) v /= dX;
    if (k == 9) v /= dY;
    if (k == 10) v = 0.125 * (red[10][0] / dY + red[11][0] / dX);
    out[k] = v / (k == 2 ? div_xy : k < 4 ? div_all : div_inner);
  }
}

}  // namespace
}  // namespace ep2d

using ep2d::fail;

extern "C" int ep2d_average_fields_noalloc(int32_t nx, int32_t ny, const double pa[EP2D_NPARS], const double* p,
                                           const double* tau_xx, const double* tau_yy, const double* tau_xy,
                                           const double* ux, const double* uy, double* out_dev, void* stream) {
  if (!pa || !p || !tau_xx || !tau_yy || !tau_xy || !ux || !uy || !out_dev)
    return fail(EP2D_ERR_ARG, "null argument");
  if (nx < 3 || ny < 3) return fail(EP2D_ERR_ARG, "the grid must be at least 3 x 3");
  if (ny - 2 > ep2d::kMaxBlocks * ep2d::kMaxRowsPerBlock)
    return fail(EP2D_ERR_ARG, "ny = " + std::to_string(ny) + " exceeds " +
                                  std::to_string(ep2d::kMaxBlocks * ep2d::kMaxRowsPerBlock + 2) +
                                  ", the largest grid the scratch-free averaging supports");
  // the checks of the library's parameter validation that concern the averaging
  for (int k = 0; k < EP2D_NPARS; k++)
    if (!std::isfinite(pa[k])) return fail(EP2D_ERR_ARG, "pa[" + std::to_string(k) + "] is not finite");
  if (!(pa[0] > 0.0) || !(pa[1] > 0.0)) return fail(EP2D_ERR_ARG, "dX and dY must be positive");
  if (!(pa[10] >= 1.0) || pa[10] > 64.0) return fail(EP2D_ERR_ARG, "N (pores per side) must be in [1, 64]");
  if (!(3.0 * pa[3] + pa[4] != 0.0)) return fail(EP2D_ERR_ARG, "3 K0 + G0 must not be zero");
  // an error left by the caller's earlier work is reported as such, not as this call's
  const cudaError_t pending = cudaPeekAtLastError();
  if (pending != cudaSuccess)
    return fail(EP2D_ERR_CUDA, std::string("a CUDA error from earlier work is pending (nothing launched): ") +
                                   cudaGetErrorString(pending));
  ep2d::AvgScratch* scratch = nullptr;
  const int rc = ep2d::scratch_on_current_device(&scratch);
  if (rc) return rc;
  // host scalars as the reference computes them (EffPlast2D.cu:453-454, :1569)
  const long nX = nx, nY = ny;
  const double K0 = pa[3], G0 = pa[4], nPores = pa[10];
  const double nu0 = (1.5 * K0 - G0) / (3.0 * K0 + G0);
  const int perOffsetX = static_cast<int>(nX / nPores);
  const int perOffsetY = static_cast<int>(nY / nPores);
  const double div_all = static_cast<double>(nX * nY);
  const double div_xy = static_cast<double>((nX - 1) * (nY - 1));
  const double div_inner = static_cast<double>((nX - 2 * perOffsetX) * (nY - 2 * perOffsetY));
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  static std::atomic<unsigned> turns{0};
  // rows per block: 1 up to four blocks per SM, 2 above (1024^2 14.4 us a call with 2, 16.4 with 1;
  // 2048^2 43.7 with 2, 46.1 with 4), 4 where the partial sums' array demands it
  const int rows = ny - 2, rpb = rows <= 592 ? 1 : rows <= 2 * ep2d::kMaxBlocks ? 2 : ep2d::kMaxRowsPerBlock;
  ep2d::k_average_reference_layout<<<(rows + rpb - 1) / rpb, ep2d::kThreads, 0, s>>>(
      nX, nY, pa[0], pa[1], p, tau_xx, tau_yy, tau_xy, ux, uy, nu0, perOffsetX, perOffsetY, rpb, div_all, div_xy,
      div_inner, scratch, turns.fetch_add(1, std::memory_order_relaxed) % ep2d::kTurns, out_dev);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return fail(EP2D_ERR_CUDA, std::string("scratch-free averaging: ") + cudaGetErrorString(e));
  return EP2D_OK;
}
