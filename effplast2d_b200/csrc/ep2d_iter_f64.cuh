// ep2d_iter_f64.cuh -- the fused iteration kernel, tile form (stress, return, update), single
// RVE and batched.
//
// One launch = one pseudo-time iteration of the reference's four kernels
// ComputeStress (EffPlast2D.cu:37-98) -> ComputeJ2 (:100-145) -> ComputePlasticity
// (:147-177) -> ComputeDisp (:3-35).  A CTA of 32 x 8 threads owns a TX x TY block of
// nodes and of the faces with the same (i, j):
//   A  stage Ux, Uy (halo 1-2) and the node mask in shared memory; the owned Vx, Vy are
//      loaded into registers at the same time, so their latency hides behind A-C;
//   B  trial stresses on the halo region: P, tauXX, tauYY at (TX+2) x (TY+2) nodes,
//      tauXY at (TX+2) x (TY+2) corners, zeroed inside pores;
//   C  (NL > 1) J2 radial return: nodes use tauXY averaged onto the node (the nine
//      edge stencils of :109-135 are one clamped 2x2 corner block), corners use tauXX,
//      tauYY averaged onto the corner, both from the pre-return values;
//   D  damped momentum update and U += V dt on the owned faces, U written to the other
//      ping-pong buffer.
// Stresses stay on chip; RECORD launches (checkpoints, last iteration) also write the
// stress fields and fold max|Vx|, max|Vy| into vmax (the convergence norm).
//
// Arithmetic: displacements and all arithmetic are FP64; velocities are stored as TV
// (double on the plain path, float on the mixed path: velocities only scale the next
// displacement increment, so their FP32 rounding is relative to a quantity that goes
// to zero and leaves no floor on the convergence test).  The per-cell formulas are
// those of ep2d_stencil.cuh, shared with the stream form, so both forms round alike.
#pragma once

#include "ep2d_stencil.cuh"
#include "ep2d_types.hpp"

namespace ep2d {

template <int TX, int TY>
struct TileSmem {
  static constexpr int UW = TX + 3, UH = TY + 3;  // Ux, Uy, mask halo tiles
  static constexpr int SW = TX + 2, SH = TY + 2;  // node stress and corner stress tiles
  static constexpr int FW = TX + 1, FH = TY + 1;  // return factors
  double ux[UH][UW];
  double uy[UH][UW];
  double p[SH][SW];
  double xx[SH][SW];
  double yy[SH][SW];
  double xy[SH][SW];
  double fn[FH][FW];
  double fc[FH][FW];
  uint8_t m[UH][UW];
};

__device__ __forceinline__ void atomic_max_nonneg(unsigned long long* addr, double v) {
  atomicMax(addr, (unsigned long long)__double_as_longlong(v));
}

// Loads of U and V.  COH (the resident form, whose grid writes the arrays it reads in
// later iterations): through L2 only (ld.global.cg), never from an SM's L1 or the
// read-only path, which do not see other SMs' stores.
template <bool COH, typename T>
__device__ __forceinline__ T ld_field(const T* p) {
  if constexpr (COH) return __ldcg(p);
  else return *p;
}

template <int TX, int TY, bool PLASTIC, bool RECORD, typename TV, bool COH = false>
__device__ __forceinline__ void iter_tile(const Geo& g, const Fields& f, const int src, const int bx, const int by,
                                          TileSmem<TX, TY>& s, bool skip = false) {
  static_assert(TX == 32 && TY % 8 == 0, "the thread mapping assumes 32 x 8 threads and TX == 32");
  using S = TileSmem<TX, TY>;
  constexpr int UW = S::UW, UH = S::UH, SW = S::SW, SH = S::SH, FW = S::FW, FH = S::FH;
  constexpr int RY = TY / 8;  // owned rows per thread

  const int tx = threadIdx.x, ty = threadIdx.y;
  const int i0 = bx * TX, j0 = by * TY;
  const int nx = g.nx, ny = g.ny;
  const size_t pitch = (size_t)g.pitch;
  const double* __restrict__ ux = src ? f.ux[1] : f.ux[0];
  const double* __restrict__ uy = src ? f.uy[1] : f.uy[0];
  double* __restrict__ uxo = src ? f.ux[0] : f.ux[1];
  double* __restrict__ uyo = src ? f.uy[0] : f.uy[1];
  TV* __restrict__ fvx = static_cast<TV*>(f.vx);
  TV* __restrict__ fvy = static_cast<TV*>(f.vy);

  // owned velocities, fetched first
  double vxr[RY], vyr[RY];
#pragma unroll
  for (int r = 0; r < RY; r++) {
    const int i = i0 + tx, j = j0 + ty + 8 * r;
    const bool ok = (i < nx && j < ny);
    vxr[r] = ok ? (double)ld_field<COH>(fvx + j * pitch + i) : 0.0;
    vyr[r] = ok ? (double)ld_field<COH>(fvy + j * pitch + i) : 0.0;
  }

  // ---- A: stage Ux (i in [i0-1, i0+TX+1], j in [j0-2, j0+TY]), Uy (i in [i0-2, i0+TX],
  //         j in [j0-1, j0+TY+1]) and the mask (nodes [i0-2, i0+TX] x [j0-2, j0+TY])
#pragma unroll
  for (int lj = ty; lj < UH; lj += 8) {
#pragma unroll
    for (int li = tx; li < UW; li += 32) {
      int i = i0 - 1 + li, j = j0 - 2 + lj;
      s.ux[lj][li] = (i >= 0 && i <= nx && j >= 0 && j < ny) ? ld_field<COH>(ux + j * pitch + i) : 0.0;
      i = i0 - 2 + li;
      j = j0 - 1 + lj;
      s.uy[lj][li] = (i >= 0 && i < nx && j >= 0 && j <= ny) ? ld_field<COH>(uy + j * pitch + i) : 0.0;
      j = j0 - 2 + lj;
      s.m[lj][li] = (i >= 0 && i < nx && j >= 0 && j < ny) ? f.mask[j * pitch + i] : (uint8_t)0;
    }
  }
  __syncthreads();

  const double rdX = g.rdX, rdY = g.rdY;
  const double third = 1.0 / 3.0;
  const double G20 = __dmul_rn(2.0, g.G0), G2p = __dmul_rn(2.0, g.Gp);
  // ---- B: trial stresses at nodes (i0-1+li, j0-1+lj) and corners (i0-2+li, j0-2+lj)
#pragma unroll
  for (int lj = ty; lj < SH; lj += 8) {
#pragma unroll
    for (int li = tx; li < SW; li += 32) {
      {
        const int i = i0 - 1 + li, j = j0 - 1 + lj;
        double pv = 0.0, xv = 0.0, yv = 0.0;
        if (i >= 0 && i < nx && j >= 0 && j < ny) {
          const uint8_t m = s.m[lj + 1][li + 1];
          if (!(m & M_NODE))
            node_trial(__dsub_rn(s.ux[lj + 1][li + 1], s.ux[lj + 1][li]), __dsub_rn(s.uy[lj + 1][li + 1], s.uy[lj][li + 1]),
                       (m & M_MAT) ? g.Kp : g.K0, (m & M_MAT) ? G2p : G20, rdX, rdY, third, pv, xv, yv);
        }
        s.p[lj][li] = pv;
        s.xx[lj][li] = xv;
        s.yy[lj][li] = yv;
      }
      {
        const int ci = i0 - 2 + li, cj = j0 - 2 + lj;
        double t = 0.0;
        if (ci >= 0 && ci < nx - 1 && cj >= 0 && cj < ny - 1) {
          const uint8_t m00 = s.m[lj][li], m10 = s.m[lj][li + 1], m01 = s.m[lj + 1][li], m11 = s.m[lj + 1][li + 1];
          if (!(m00 & M_CORNER))
            t = corner_trial(corner_g4(m00, m10, m01, m11, g.G0, g.Gp), __dsub_rn(s.ux[lj + 1][li], s.ux[lj][li]),
                             __dsub_rn(s.uy[lj][li + 1], s.uy[lj][li]), rdX, rdY);
        }
        s.xy[lj][li] = t;
      }
    }
  }
  __syncthreads();

  // ---- C: J2 radial return (NL > 1, EffPlast2D.cu:392-397)
  if (PLASTIC) {
    const double coh = g.coh, coh2 = g.coh2, coh4 = g.coh4, coh2x16 = g.coh2x16;
#pragma unroll
    for (int lj = ty; lj < FH; lj += 8) {
#pragma unroll
      for (int li = tx; li < FW; li += 32) {
        {  // node (i0-1+li, j0-1+lj)
          const int i = i0 - 1 + li, j = j0 - 1 + lj;
          double fn = 1.0;
          if (i >= 0 && i < nx && j >= 0 && j < ny) {
            const int a = min(max(i - 1, 0), nx - 3) - (i0 - 2), b = min(max(j - 1, 0), ny - 3) - (j0 - 2);
            const double hsum = pair_sum4(s.xy[b][a], s.xy[b][a + 1], s.xy[b + 1][a], s.xy[b + 1][a + 1]);
            const double xv = s.xx[lj][li], yv = s.yy[lj][li];
            const double J2sq = node_j2sq_h(xv, yv, hsum);
            fn = return_factor(J2sq, coh, coh2);
            if (RECORD && li >= 1 && lj >= 1) {
              const double tavo = __dmul_rn(__dmul_rn(0.25, hsum), fn);
              const double J2o =
                  (fn != 1.0) ? __dsqrt_rn(node_j2sq(__dmul_rn(xv, fn), __dmul_rn(yv, fn), tavo)) : __dsqrt_rn(J2sq);
              f.txyav[j * pitch + i] = tavo;
              f.j2[j * pitch + i] = J2o;
            }
          }
          s.fn[lj][li] = fn;
        }
        {  // corner (i0-1+li, j0-1+lj)
          const int ci = i0 - 1 + li, cj = j0 - 1 + lj;
          double fc = 1.0;
          if (ci >= 0 && ci < nx - 1 && cj >= 0 && cj < ny - 1) {
            // column pairs: nodes (i, j) + (i, j+1), then (i+1, j) + (i+1, j+1)
            const double sx = pair_sum4(s.xx[lj][li], s.xx[lj + 1][li], s.xx[lj][li + 1], s.xx[lj + 1][li + 1]);
            const double sy = pair_sum4(s.yy[lj][li], s.yy[lj + 1][li], s.yy[lj][li + 1], s.yy[lj + 1][li + 1]);
            const double J2sq16 = corner_j2sq16(sx, sy, s.xy[lj + 1][li + 1]);  // 16 J2^2
            fc = return_factor(J2sq16, coh4, coh2x16);
            if (RECORD && li >= 1 && lj >= 1) f.j2xy[cj * pitch + ci] = __dmul_rn(0.25, __dsqrt_rn(J2sq16));
          }
          s.fc[lj][li] = fc;
        }
      }
    }
    __syncthreads();
#pragma unroll
    for (int lj = ty; lj < FH; lj += 8) {
#pragma unroll
      for (int li = tx; li < FW; li += 32) {
        const double fn = s.fn[lj][li];
        s.xx[lj][li] = __dmul_rn(s.xx[lj][li], fn);
        s.yy[lj][li] = __dmul_rn(s.yy[lj][li], fn);
        s.xy[lj + 1][li + 1] = __dmul_rn(s.xy[lj + 1][li + 1], s.fc[lj][li]);
      }
    }
    __syncthreads();
  }

  if (skip) return;  // all threads

  // ---- D: damped momentum update and U += V dt on the owned faces
  const double dT = g.dT, cX = g.cX, cY = g.cY, dtrX = g.dtrX, dtrY = g.dtrY;
  double vmx = 0.0, vmy = 0.0;
#pragma unroll
  for (int r = 0; r < RY; r++) {
    const int li = tx, lj = ty + 8 * r;
    const int i = i0 + li, j = j0 + lj;
    if (i >= nx || j >= ny) continue;
    const size_t q = j * pitch + i;
    double vx = vxr[r];
    if (i > 0 && j > 0 && j < ny - 1) {
      vx = face_velocity_s(vx, cX,
                           stress_diff(s.p[lj + 1][li + 1], s.p[lj + 1][li], s.xx[lj + 1][li + 1], s.xx[lj + 1][li]),
                           dtrX, __dsub_rn(s.xy[lj + 2][li + 1], s.xy[lj + 1][li + 1]), dtrY);
      const TV vs = (TV)vx;
      fvx[q] = vs;
      vx = (double)vs;  // the displacement moves by the stored velocity
    }
    uxo[q] = advance(s.ux[lj + 2][li + 1], vx, dT);
    double vy = vyr[r];
    if (i > 0 && i < nx - 1 && j > 0) {
      vy = face_velocity_s(vy, cY,
                           stress_diff(s.p[lj + 1][li + 1], s.p[lj][li + 1], s.yy[lj + 1][li + 1], s.yy[lj][li + 1]),
                           dtrY, __dsub_rn(s.xy[lj + 1][li + 2], s.xy[lj + 1][li + 1]), dtrX);
      const TV vs = (TV)vy;
      fvy[q] = vs;
      vy = (double)vs;
    }
    uyo[q] = advance(s.uy[lj + 1][li + 2], vy, dT);
    if (i == nx - 1) {  // face column i = nx of Ux/Vx: never updated by the reference
      const size_t q2 = j * pitch + nx;
      uxo[q2] = s.ux[lj + 2][li + 2];
      if (RECORD) vmx = fmax(vmx, fabs((double)fvx[q2]));
    }
    if (j == ny - 1) {  // face row j = ny of Uy/Vy
      const size_t q3 = (size_t)ny * pitch + i;
      uyo[q3] = s.uy[lj + 2][li + 2];
      if (RECORD) vmy = fmax(vmy, fabs((double)fvy[q3]));
    }
    if (RECORD) {
      vmx = fmax(vmx, fabs(vx));
      vmy = fmax(vmy, fabs(vy));
      f.p[q] = s.p[lj + 1][li + 1];
      f.txx[q] = s.xx[lj + 1][li + 1];
      f.tyy[q] = s.yy[lj + 1][li + 1];
      if (i < nx - 1 && j < ny - 1) f.txy[q] = s.xy[lj + 2][li + 2];
    }
  }
  if (RECORD) {
    for (int o = 16; o > 0; o >>= 1) {
      vmx = fmax(vmx, __shfl_xor_sync(0xffffffffu, vmx, o));
      vmy = fmax(vmy, __shfl_xor_sync(0xffffffffu, vmy, o));
    }
    if (tx == 0) {
      atomic_max_nonneg(&f.vmax[0], vmx);
      atomic_max_nonneg(&f.vmax[1], vmy);
    }
  }
}

// An on-chip launch has given up (CHIP_GAVE_UP): the recording launch behind it leaves the state
// alone (U and V; the stresses it is there to write anew), and the host runs the interval again.
__device__ __forceinline__ bool chip_failed(const Fields& f) {
  return (*reinterpret_cast<const volatile unsigned*>(f.gbar + 3) & CHIP_FAILED) != 0;
}

// One RVE: one CTA per tile.
template <int TX, int TY, bool PLASTIC, bool RECORD, typename TV>
__global__ void __launch_bounds__(256) k_iter(Geo g, Fields f, int src) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const bool skip = RECORD && chip_failed(f);
  iter_tile<TX, TY, PLASTIC, RECORD, TV>(g, f, src, blockIdx.x, blockIdx.y,
                                         *reinterpret_cast<TileSmem<TX, TY>*>(smem_raw), skip);
}

// Many RVEs: a persistent grid walks the device-side tile list {rve, bx | by << 16}.
// The list and its length live in device memory, so a captured graph of these
// launches stays valid while RVEs join and retire; `parity` is the launch's position
// in the graph (mod 2), flipping every RVE's ping-pong buffers in lockstep.
template <int TX, int TY, bool RECORD, typename TV>
__global__ void __launch_bounds__(256) k_iter_batch(const BatchEntry* __restrict__ ents, const int2* __restrict__ tiles,
                                                    const int* __restrict__ ntiles, int parity) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  TileSmem<TX, TY>& s = *reinterpret_cast<TileSmem<TX, TY>*>(smem_raw);
  const int n = *ntiles;
  for (int t = blockIdx.x; t < n; t += gridDim.x) {
    const int2 tc = tiles[t];
    const BatchEntry& e = ents[tc.x];
    const int src = e.src0 ^ parity;
    if (e.plastic) iter_tile<TX, TY, true, RECORD, TV>(e.g, e.f, src, tc.y & 0xffff, tc.y >> 16, s);
    else iter_tile<TX, TY, false, RECORD, TV>(e.g, e.f, src, tc.y & 0xffff, tc.y >> 16, s);
    __syncthreads();  // shared memory is reused by the next tile
  }
}

// ---- resident form: many iterations per launch ---------------------------------------
// The reference launches its four kernels once per iteration with a device-wide sync
// after each (EffPlast2D.cu:389-399); the per-launch forms fuse them into one launch per
// iteration.  On grids too small to fill the GPU (a few hundred cells per SM) an
// iteration is a few microseconds of work, and the launch boundary is a large part of
// it.  The resident form runs all the iterations between two checkpoints in ONE
// cooperative launch: every CTA stays resident, owns fixed tiles, and after each
// iteration meets the others at a grid-wide barrier (the iteration's U is then complete
// and visible, and the next one reads it).  Per tile it runs iter_tile, so its results
// equal the tile form's bit for bit.
//
// The barrier lives in device memory (`Fields::gbar`): gbar[0..1] is a 64-bit count of
// arrivals, zeroed by the host before each launch; gbar[2] is an error flag, zero when
// the RVE is created or reset.  Barrier k (k = 1, 2, ...) of a launch is passed
// once the count reaches k x gridDim.x: each CTA adds 1 with release semantics after
// its threads' stores (a CTA barrier first) and one thread polls the count with acquire
// semantics (a CTA barrier after), the pattern of a semaphore between CTAs; the count
// is never reset within a launch, so there is no generation to track.  Every wait is
// bounded: a CTA that waits longer than timeout_ns sets the flag and returns, and a CTA
// that sees the flag returns too, so a barrier that cannot complete ends the launch with
// the flag set instead of hanging.  The flag stays set until the RVE is reset (later launches return at
// once); the host reads it at every checkpoint and reports the RVE as failed.

__device__ __forceinline__ unsigned long long ld_acquire_u64(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

// true once the arrival count reaches `target`; false if the wait ran out or another
// CTA's did
__device__ __forceinline__ bool grid_barrier(unsigned* gbar, unsigned long long target,
                                             unsigned long long timeout_ns, int* s_ok) {
  __syncthreads();  // the CTA's stores of this iteration are issued
  if (threadIdx.x == 0 && threadIdx.y == 0) {
    unsigned long long* cnt = reinterpret_cast<unsigned long long*>(gbar);
    asm volatile("red.release.gpu.global.add.u64 [%0], 1;" ::"l"(cnt) : "memory");
    int ok = 1;
    if (ld_acquire_u64(cnt) < target) {
      const unsigned long long t0 = global_ns();
      for (;;) {
        __nanosleep(32);
        if (ld_acquire_u64(cnt) >= target) break;
        if (*reinterpret_cast<volatile unsigned*>(gbar + 2)) {
          ok = 0;
          break;
        }
        if (global_ns() - t0 > timeout_ns) {
          atomicExch(&gbar[2], 1u);
          ok = 0;
          break;
        }
      }
    }
    *s_ok = ok;
  }
  __syncthreads();  // the other CTAs' stores are visible to this CTA's later loads
  return *s_ok != 0;
}

// n_iter plain iterations (no recording) of one RVE, starting from buffer src0.  The
// grid is 1-D and co-resident (cooperative launch); CTA b owns tiles b, b + grid, ...
template <int TX, int TY, bool PLASTIC, typename TV>
__global__ void __launch_bounds__(256) k_iter_resident(Geo g, Fields f, int src0, int n_iter,
                                                       unsigned long long timeout_ns) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int s_ok;
  TileSmem<TX, TY>& s = *reinterpret_cast<TileSmem<TX, TY>*>(smem_raw);
  const int ntx = (g.nx + TX - 1) / TX, nty = (g.ny + TY - 1) / TY;
  const int ntiles = ntx * nty;
  if (*reinterpret_cast<volatile unsigned*>(f.gbar + 2)) return;  // an earlier launch failed
  for (int it = 0; it < n_iter; it++) {
    const int src = src0 ^ (it & 1);
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
      iter_tile<TX, TY, PLASTIC, false, TV, true>(g, f, src, t % ntx, t / ntx, s);
      __syncthreads();  // shared memory is reused by the next tile
    }
    if (it + 1 < n_iter &&
        !grid_barrier(f.gbar, (unsigned long long)(it + 1) * gridDim.x, timeout_ns, &s_ok))
      return;
  }
}

// The barrier alone, for the host's check of its failure path: `missing` of the grid's
// CTAs never arrive (they return at once), so with missing > 0 the others' waits run
// out after timeout_ns and the flag is set; with missing == 0 every round completes.
// out[0] = CTAs that passed all rounds.
__global__ void k_grid_barrier_check(unsigned* gbar, int missing, int rounds, unsigned long long timeout_ns,
                                     unsigned* out) {
  __shared__ int s_ok;
  if ((int)blockIdx.x < missing) return;
  for (int r = 0; r < rounds; r++)
    if (!grid_barrier(gbar, (unsigned long long)(r + 1) * gridDim.x, timeout_ns, &s_ok)) return;
  if (threadIdx.x == 0 && threadIdx.y == 0) atomicAdd(out, 1u);
}

}  // namespace ep2d
