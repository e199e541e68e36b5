// ep2d_iter_chip.cuh -- the fused iteration kernel, on-chip form: a run of plain
// iterations of one RVE in one launch, the state held on the SMs throughout.
//
// Same iteration as the other forms (ComputeStress -> ComputeJ2 -> ComputePlasticity ->
// ComputeDisp, EffPlast2D.cu:3-177) and the same per-cell formulas (ep2d_stencil.cuh), so
// its results equal theirs bit for bit.  A CTA owns a tile of STREAM_COLS columns x
// (warps x R) rows; each warp marches up its R rows as the stream form does (lanes = 28
// owned columns and 2 halo columns on each side, neighbours by shuffles), two rows per
// step.  U of the tile and its 2-wide halo lives in shared memory, V in tensor memory
// (every lane's own column of its warp's rows: a private 512-byte-per-lane store that
// costs neither registers nor shared-memory bandwidth), and only the tile's 2-wide rim of
// U leaves the SM each iteration.
//
// The rim goes to the neighbouring CTAs through L2 as 16-byte records {lo, tag, hi, tag}
// of a double, tag = the iteration: a reader polls the record itself until both tags are
// the iteration's, so one L2 round trip both carries the value and synchronises, with no
// fence, flag or grid-wide barrier (each 8-byte half {word, tag} is written by one
// vector store and is valid on its own).  Records are double-buffered by iteration parity: a CTA
// overwrites iteration t's records in iteration t + 2, after it has read its neighbours'
// records of t + 1, which they wrote after reading all of t's.  Waits are bounded: a CTA that
// waits longer than timeout_ns sets its RVE's error flag and leaves, the others
// follow, and the host reports the RVE as failed.
//
// Within a CTA the two lowest and two highest rows of a warp are read by the warps below
// and above and are double-buffered by parity; the rows between are updated in place.
// One barrier of the tile's warps per iteration.  All CTAs must be resident at once
// (cooperative launch, one CTA per SM).
//
// What bounds it: on grids up to ~400^2 latency, the rim exchange (1.4 us of an iteration
// with the march left out) and one warp's march; on larger ones the issue of the march's
// instructions.  Measured, us per iteration, the form the library took before / this one
// (FP64): elastic 128^2 4.2 / 1.74, 512^2 6.3 / 2.53, 1024^2 15.5 / 5.7; with the return map
// 128^2 5.8 / 2.41, 256^2 6.2 / 2.70, 512^2 8.9 / 4.27, 768^2 14.3 / 6.85, 1024^2 16.3 / 9.9.
#pragma once

#include "ep2d_iter_f64.cuh"
#include "ep2d_iter_stream.cuh"
#include "ep2d_stencil.cuh"
#include "ep2d_types.hpp"

namespace ep2d {

// material constants of a node and a corner, by the 7-bit index of chip_index
struct __align__(16) ChipMat {
  double k, g2, g4, pad;
};
constexpr int CHIP_MATS = 128;
// row pairs per turn of the march's loop: 2 measured best (1024^2, 16 rows: 9.85 us an
// iteration; 1: 10.5, 4: 9.94 with spills)
constexpr int kChipUnroll = 2;

// shared memory, in bytes: materials, U rows (32 columns of (Ux, Uy)) in pairs, the material
// index of every (row, column), and the poll list
constexpr int CHIP_ROW = 32 * 16, CHIP_PAIR = 2 * CHIP_ROW;
__host__ __device__ constexpr int chip_pairs_per_warp(int rows) { return rows == 2 ? 2 : rows / 2 + 2; }
// cells a lane polls: of the columns beside its warp's rows (4 per row), of the rows below
// and above the tile (2 x 2 x 32 cells, spread over the group's warps)
__host__ __device__ constexpr int chip_col_polls(int rows) { return (4 * rows + 31) / 32; }
__host__ __device__ constexpr int chip_polls(int warps, int rows) {
  return chip_col_polls(rows) + (4 + warps - 1) / warps;
}
__host__ __device__ constexpr size_t chip_group_bytes(int warps, int rows) {
  return (size_t)(warps * chip_pairs_per_warp(rows) + 4) * CHIP_PAIR + (size_t)(warps * rows + 4) * 32 +
         (size_t)warps * chip_polls(warps, rows) * 32 * sizeof(uint2);
}
// with tracking, a byte of yield bits per (row, column) behind the groups' regions
__host__ __device__ constexpr size_t chip_smem_bytes(int groups, int warps, int rows, bool track = false) {
  return CHIP_MATS * sizeof(ChipMat) + groups * (chip_group_bytes(warps, rows) + (track ? warps * rows * 32 : 0));
}

// barrier of one group's threads that also ORs a flag over them
__device__ __forceinline__ bool group_barrier_or(int id, int threads, int flag) {
  int r;
  asm volatile(
      "{\n .reg .pred p, q;\n setp.ne.s32 p, %1, 0;\n barrier.cta.red.or.pred q, %2, %3, p;\n"
      " selp.s32 %0, 1, 0, q;\n}"
      : "=r"(r)
      : "r"(flag), "r"(id), "r"(threads)
      : "memory");
  return r != 0;
}

// index of the material constants of node (i, r) and corner (i, r): bits 0-1 the node's
// M_MAT | M_NODE, bits 2-6 the corner's corner_index.  A node outside the grid counts as
// a pore node and a corner outside it as a pore corner: their stresses are 0.
__device__ __forceinline__ int chip_index(const Geo& g, const uint8_t* mask, int i, int r) {
  const bool node = i >= 0 && i < g.nx && r >= 0 && r < g.ny;
  const bool corner = i >= 0 && i < g.nx - 1 && r >= 0 && r < g.ny - 1;
  const int m = node ? mask[r * g.pitch + i] : (int)M_NODE;
  const int up = corner ? mask[(r + 1) * g.pitch + i] : 0;
  return (m & (M_MAT | M_NODE)) | ((corner ? corner_index(m, up) : (int)M_CORNER) << 2);
}

// ---- tensor memory: private words of a lane -------------------------------------------
__device__ __forceinline__ void tmem_ld(uint32_t addr, uint32_t (&v)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
               : "r"(addr));
}
__device__ __forceinline__ void tmem_ld(uint32_t addr, uint32_t (&v)[4]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3])
               : "r"(addr));
}
// the loaded registers pass through the wait, so no use of them can move above it
__device__ __forceinline__ void tmem_ld_wait(uint32_t (&v)[8]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]));
}
__device__ __forceinline__ void tmem_ld_wait(uint32_t (&v)[4]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;" : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]));
}
__device__ __forceinline__ void tmem_st(uint32_t addr, const uint32_t (&v)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(addr), "r"(v[0]),
               "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]));
}
__device__ __forceinline__ void tmem_st(uint32_t addr, const uint32_t (&v)[4]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(v[0]), "r"(v[1]),
               "r"(v[2]), "r"(v[3]));
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// (vx, vy) of two rows as the words of a pair, and back
template <typename TV>
struct VPair;
template <>
struct VPair<double> {
  uint32_t w[8];
  __device__ double get(int k) const { return __hiloint2double((int)w[2 * k + 1], (int)w[2 * k]); }
  __device__ void set(int k, double v) {
    w[2 * k] = (uint32_t)__double2loint(v);
    w[2 * k + 1] = (uint32_t)__double2hiint(v);
  }
};
template <>
struct VPair<float> {
  uint32_t w[4];
  __device__ float get(int k) const { return __uint_as_float(w[k]); }
  __device__ void set(int k, float v) { w[k] = __float_as_uint(v); }
};

// ---- rim records ------------------------------------------------------------------------
// Record of a cell: {lo, tag, hi, tag} of Ux and of Uy, one 256-bit access.
struct RimRecord {
  uint32_t w[8];
  __device__ bool ready(uint32_t tag) const { return ((w[1] ^ tag) | (w[3] ^ tag) | (w[5] ^ tag) | (w[7] ^ tag)) == 0; }
  __device__ double2 value() const {
    return make_double2(__hiloint2double((int)w[2], (int)w[0]), __hiloint2double((int)w[6], (int)w[4]));
  }
};
constexpr int RIM_BYTES = 32;
// records a lane has in flight while it polls: 2 (3 and 4 cost the march registers, 128 being
// all there are: 1024^2 9.85 -> 10.6 us an iteration)
constexpr int kRimInFlight = 2;
__device__ __forceinline__ void rim_put(char* rec, const double2& u, uint32_t tag) {
  asm volatile("st.relaxed.gpu.global.v8.b32 [%0], {%1,%5,%2,%5,%3,%5,%4,%5};" ::"l"(rec), "r"(__double2loint(u.x)),
               "r"(__double2hiint(u.x)), "r"(__double2loint(u.y)), "r"(__double2hiint(u.y)), "r"(tag)
               : "memory");
}
__device__ __forceinline__ void rim_get(const char* rec, RimRecord& r) {
  asm volatile("ld.relaxed.gpu.global.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r.w[0]), "=r"(r.w[1]), "=r"(r.w[2]), "=r"(r.w[3]), "=r"(r.w[4]), "=r"(r.w[5]), "=r"(r.w[6]),
                 "=r"(r.w[7])
               : "l"(rec)
               : "memory");
}

// where a warp's row pairs lie: pair q of its rows/2, copy `par` of the double-buffered ones
__device__ __forceinline__ uint32_t chip_pair_off(int q, int npairs, int par) {
  if (q == 0) return par * CHIP_PAIR;
  if (q == npairs - 1) return (2 + par) * CHIP_PAIR;
  return (3 + q) * CHIP_PAIR;
}

// One iteration of one warp's rows jA .. jA + 2 npairs - 1 (copy `par` to copy par ^ 1).
// rd0 / rdN: the row pairs below and above the warp's own; idx: material indices of row
// jA - 2 on, 32 per row; vmem: tensor-memory address of the warp's V.
// NP: the number of row pairs where it is known (1 to 3: the march unrolled, so that its rows'
// chains overlap: 256^2, 2 rows, 2.70 -> 2.54 us an iteration; 448^2, 4 rows, 3.76 -> 3.55; 512^2, 6
// rows, 4.29 -> 4.07), else 0.
template <bool PLASTIC, bool EDGE, int NP, typename TV, bool TRACK>
__device__ __forceinline__ void chip_march(const Geo& g, const ChipMat* __restrict__ mats, const uint8_t* idx,
                                           const char* rd0, char* own, const char* rdN, int npairs_in, int par, int i,
                                           int jA, uint32_t vmem, uint8_t* yielded) {
  constexpr int VW = sizeof(VPair<TV>) / 4;
  const int npairs = NP ? NP : npairs_in;
  const int lane = threadIdx.x & 31;
  const int nx = g.nx, ny = g.ny;
  const int right = lane < 31 ? 1 : 0;
  const bool col_own = lane >= 2 && lane < 2 + STREAM_COLS && (!EDGE || i < nx);
  const double rdX = g.rdX, rdY = g.rdY, third = 1.0 / 3.0;
  const double coh = g.coh, coh2 = g.coh2, coh4 = g.coh4, coh2x16 = g.coh2x16;
  const double dT = g.dT, cX = g.cX, cY = g.cY, dtrX = g.dtrX, dtrY = g.dtrY;
  int sa = 0, sb = 0;  // lanes of the node's clamped corner columns
  if (EDGE) {
    const int a = min(max(i - 1, 0), nx - 3) - i;
    sa = min(max(lane + a, 0), 31);
    sb = min(max(lane + a + 1, 0), 31);
  }

  double uxc = 0, uxc_r = 0, uyc = 0;             // U of the last row read
  double pb = 0, xb = 0, yb = 0, cb = 0;          // trial stresses of the last row
  double hz = 0, h0 = 0, h1 = 0;                  // corner pair sums of the last three rows
  double syq = 0, cq = 0, cq_l = 0;               // returned: total syy, corner of the row below
  const char* rd_prev = rd0;

  auto corner_pair = [&](double c) {
    return EDGE ? add_rn(shfl_idx(c, sa), shfl_idx(c, sb)) : add_rn(shfl_up1(c), c);
  };
  // 4-corner sum of node row j from the pair sums of corner rows j - 2 .. j + 1
  auto corner_sum = [&](int j, double hm2, double hm1, double hj, double hp1) {
    if (EDGE) return j == 0 ? add_rn(hj, hp1) : j == ny - 1 ? add_rn(hm2, hm1) : add_rn(hm1, hj);
    return add_rn(hm1, hj);
  };
  // 16 J2^2 of a corner of row j from the node deviators of rows j and j + 1
  auto corner_j2 = [&](double x, double y, double c, double xn, double yn) {
    const double vx = add_rn(x, xn), vy = add_rn(y, yn);
    const double tx = add_rn(vx, shfl_dn(vx)), ty = add_rn(vy, shfl_dn(vy));
    return corner_j2sq16(tx, ty, c);
  };
  // return_factor without a branch of its own: rsqrt of a value that is always in range
  auto factor = [&](double j2, double lim2, double lim) {
    const bool yields = j2 > lim2;
    const double r = mul_rn(lim, rsqrt(yields ? j2 : lim2));
    return yields ? r : 1.0;
  };
  // faces of row j: new velocities and displacements from the old ones
  auto face = [&](int j, double sx, double sx_l, double sy, double cw_l, TV& vx, TV& vy, double2& u) {
    const double vxo = (double)vx, vyo = (double)vy;
    const TV vxs = (TV)face_velocity_s(vxo, cX, sub_rn(sx, sx_l), dtrX, sub_rn(cw_l, cq_l), dtrY);
    const TV vys = (TV)face_velocity_s(vyo, cY, sub_rn(sy, syq), dtrY, sub_rn(cq, cq_l), dtrX);
    if (EDGE) {
      if (i > 0 && j > 0 && j < ny - 1) vx = vxs;
      if (i > 0 && i < nx - 1 && j > 0) vy = vys;
    } else {
      vx = vxs;
      vy = vys;
    }
    u.x = advance(u.x, (double)vx, dT);
    u.y = advance(u.y, (double)vy, dT);
  };

  auto pair = [&](auto stage_c, int p, const char* rd, char* wr) {
    constexpr int STAGE = decltype(stage_c)::value;
    // the other lanes have read the rows this step overwrites (with one or two pairs every
    // row is double-buffered)
    if (NP == 0 || NP > 2) __syncwarp();
    VPair<TV> v;
    if constexpr (STAGE == 2) tmem_ld(vmem + (p - 2) * VW, v.w);
    const double2* ra = reinterpret_cast<const double2*>(rd) + lane;
    const double2 ua = ra[0], uar = ra[right], ub = ra[32], ubr = ra[32 + right];
    const uint8_t* ip = idx + (2 * p) * 32 + lane;  // row ka
    double p1 = 0, x1 = 0, y1 = 0, c1 = 0, p2, x2, y2, c2, hs1 = 0, hs2 = 0;
    if constexpr (STAGE >= 1) {  // trial of row ka - 1
      const ChipMat& m = mats[ip[-32]];
      node_trial(sub_rn(uxc_r, uxc), sub_rn(ua.y, uyc), m.k, m.g2, rdX, rdY, third, p1, x1, y1);
      c1 = corner_trial(m.g4, sub_rn(uar.x, uxc_r), sub_rn(uar.y, ua.y), rdX, rdY);
      if (PLASTIC) hs1 = corner_pair(c1);
    }
    {  // trial of row ka
      const ChipMat& m = mats[ip[0]];
      node_trial(sub_rn(uar.x, ua.x), sub_rn(ub.y, ua.y), m.k, m.g2, rdX, rdY, third, p2, x2, y2);
      c2 = corner_trial(m.g4, sub_rn(ubr.x, uar.x), sub_rn(ubr.y, ub.y), rdX, rdY);
      if (PLASTIC) hs2 = corner_pair(c2);
    }
    const int ja = jA + 2 * p - 4;  // row ka - 2
    if constexpr (STAGE == 2) {
      const double2* uo = reinterpret_cast<const double2*>(rd_prev) + lane;
      double2 u0 = uo[0], u1 = uo[32];
      double xr0 = xb, yr0 = yb, cw0 = cb, xr1 = x1, yr1 = y1, cw1 = c1;
      if (PLASTIC) {
        const double n0 = node_j2sq_h(xb, yb, corner_sum(ja, hz, h0, h1, hs1));
        const double n1 = node_j2sq_h(x1, y1, corner_sum(ja + 1, h0, h1, hs1, hs2));
        const double m0 = corner_j2(xb, yb, cb, x1, y1), m1 = corner_j2(x1, y1, c1, x2, y2);
        if (__any_sync(0xffffffffu, n0 > coh2 || n1 > coh2 || m0 > coh2x16 || m1 > coh2x16)) {
          const double f0 = factor(n0, coh2, coh), f1 = factor(n1, coh2, coh);
          xr0 = mul_rn(xb, f0);
          yr0 = mul_rn(yb, f0);
          cw0 = mul_rn(cb, factor(m0, coh2x16, coh4));
          xr1 = mul_rn(x1, f1);
          yr1 = mul_rn(y1, f1);
          cw1 = mul_rn(c1, factor(m1, coh2x16, coh4));
          if (TRACK) {  // J2 > coh from the trial stresses (get_sigma_2D.m:126-138); a corner inside the grid
            uint8_t* yl = yielded + 2 * (p - 2) * 32 + lane;
            const bool c_in = !EDGE || i < nx - 1;
            const int b0 = (n0 > coh2 ? M_YN : 0) | (c_in && (!EDGE || ja < ny - 1) && m0 > coh2x16 ? M_YC : 0);
            const int b1 = (n1 > coh2 ? M_YN : 0) | (c_in && (!EDGE || ja + 1 < ny - 1) && m1 > coh2x16 ? M_YC : 0);
            yl[0] |= b0;
            yl[32] |= b1;
          }
        }
      }
      const double sx0 = sub_rn(xr0, pb), sy0 = sub_rn(yr0, pb), sx1 = sub_rn(xr1, p1), sy1 = sub_rn(yr1, p1);
      const double cw0_l = shfl_up1(cw0), sx0_l = shfl_up1(sx0);
      const double cw1_l = shfl_up1(cw1), sx1_l = shfl_up1(sx1);
      tmem_ld_wait(v.w);
      TV v0x = v.get(0), v0y = v.get(1), v1x = v.get(2), v1y = v.get(3);
      face(ja, sx0, sx0_l, sy0, cw0_l, v0x, v0y, u0);
      syq = sy0;
      cq = cw0;
      cq_l = cw0_l;
      face(ja + 1, sx1, sx1_l, sy1, cw1_l, v1x, v1y, u1);
      syq = sy1;
      cq = cw1;
      cq_l = cw1_l;
      v.set(0, v0x);
      v.set(1, v0y);
      v.set(2, v1x);
      v.set(3, v1y);
      tmem_st(vmem + (p - 2) * VW, v.w);
      double2* un = reinterpret_cast<double2*>(wr) + lane;
      if (col_own && (!EDGE || ja < ny)) un[0] = u0;
      if (col_own && (!EDGE || ja + 1 < ny)) un[32] = u1;
    } else if constexpr (STAGE == 1) {
      double yr = y1;
      cq = c1;
      if (PLASTIC) {
        yr = mul_rn(y1, factor(node_j2sq_h(x1, y1, corner_sum(ja + 1, h0, h1, hs1, hs2)), coh2, coh));
        cq = mul_rn(c1, factor(corner_j2(x1, y1, c1, x2, y2), coh2x16, coh4));
      }
      syq = sub_rn(yr, p1);
      cq_l = shfl_up1(cq);
    }
    uxc = ub.x;
    uxc_r = ubr.x;
    uyc = ub.y;
    pb = p2;
    xb = x2;
    yb = y2;
    cb = c2;
    hz = h1;
    h0 = hs1;
    h1 = hs2;
    rd_prev = rd;
  };
  pair(std::integral_constant<int, 0>{}, 0, rd0, nullptr);
  pair(std::integral_constant<int, 1>{}, 1, own + chip_pair_off(0, npairs, par), nullptr);
#pragma unroll (NP ? NP : kChipUnroll)
  for (int p = 2; p <= npairs + 1; p++)
    pair(std::integral_constant<int, 2>{}, p, p <= npairs ? own + chip_pair_off(p - 1, npairs, par) : rdN,
         own + chip_pair_off(p - 2, npairs, par ^ 1));
  tmem_st_wait();
}

// a.n_iter plain iterations of every job's RVE from its buffer `src`, ending in buffer
// src ^ (n_iter & 1) (n_iter >= 2: when the buffers coincide, a tile is written back only after
// its neighbours have read it).  CTAs of groups of a.warps warps, a group per tile, a.rows rows per
// warp.  rim: records [2][tile][4 H + 112 cells].  PLASTIC 0, 1: all jobs; 2: per job.
// TRACK: also mark the nodes and corners that yield at any of the iterations (M_YN, M_YC).
template <int PLASTIC, int JOBS, typename TV, bool TRACK = false>
__global__ void __launch_bounds__(32 * CHIP_WARPS, 1) k_iter_chip(const __grid_constant__ ChipArgs<JOBS> a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ uint32_t s_tmem;
  int jb = 0;
  if (JOBS > 1)
    while (jb + 1 < a.njobs && (int)blockIdx.x >= a.job[jb + 1].cta0) jb++;
  const ChipJob& job = a.job[jb];
  const Geo& g = job.g;
  const Fields& f = job.f;
  const int nw = a.warps, rows = a.rows, n_iter = a.n_iter, ncx = job.ncx, ncy = job.ncy, src = job.src;
  const int lane = threadIdx.x & 31, wc = threadIdx.x >> 5;  // warp of the CTA
  const int group = wc / nw, w = wc - group * nw;             // its group, warp of the group
  const int groups = (int)(blockDim.x >> 5) / nw;
  const int tile = ((int)blockIdx.x - job.cta0) * groups + group;
  const bool idle = tile >= ncx * ncy;
  const int cx = tile % ncx, cy = tile / ncx;
  const int nx = g.nx, ny = g.ny, pitch = g.pitch;
  const int H = nw * rows, x0 = STREAM_COLS * cx, y0 = H * cy;
  const int npairs = rows / 2, ppw = chip_pairs_per_warp(rows);
  const int ncol = chip_col_polls(rows), npoll = chip_polls(nw, rows);
  if (__syncthreads_or(*reinterpret_cast<volatile unsigned*>(job.flag) != 0)) return;  // an earlier launch failed

  ChipMat* mats = reinterpret_cast<ChipMat*>(smem_raw);
  char* urows = reinterpret_cast<char*>(smem_raw) + CHIP_MATS * sizeof(ChipMat) + group * chip_group_bytes(nw, rows);
  char* halo_b = urows + nw * ppw * CHIP_PAIR;
  char* halo_t = halo_b + 2 * CHIP_PAIR;  // the rows below and above the tile, two copies each
  uint8_t* idx = reinterpret_cast<uint8_t*>(halo_t + 2 * CHIP_PAIR);
  uint2* polls = reinterpret_cast<uint2*>(idx + (H + 4) * 32);
  uint8_t* yielded = smem_raw + chip_smem_bytes(groups, nw, rows) + wc * rows * 32;  // TRACK only

  if (wc == 0) {  // one CTA per SM takes all of the SM's tensor memory
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(
                     (uint32_t)__cvta_generic_to_shared(&s_tmem))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  for (int t = threadIdx.x; t < CHIP_MATS; t += blockDim.x) {
    ChipMat m{0.0, 0.0, g4z_entry(t >> 2, g.G0, g.Gp), 0.0};
    if (!(t & M_NODE)) {
      m.k = (t & M_MAT) ? g.Kp : g.K0;
      m.g2 = __dmul_rn(2.0, (t & M_MAT) ? g.Gp : g.G0);
    }
    mats[t] = m;
  }
  __syncthreads();
  if (!idle) {
    const int i = x0 - 2 + lane;
    const int jA = y0 + w * rows;
    for (int r = w; r < H + 3; r += nw) idx[r * 32 + lane] = (uint8_t)chip_index(g, f.mask, i, y0 - 2 + r);

    // U of the tile and its halo, both copies of the double-buffered rows (faces outside the
    // arrays: 0; the face column nx of Ux and row ny of Uy never change)
    const double* __restrict__ ux = f.ux[src];
    const double* __restrict__ uy = f.uy[src];
    auto load_u = [&](int j) {
      double2 u;
      u.x = (i >= 0 && i <= nx && j >= 0 && j < ny) ? ux[j * pitch + i] : 0.0;
      u.y = (i >= 0 && i < nx && j >= 0 && j <= ny) ? uy[j * pitch + i] : 0.0;
      return u;
    };
    char* own = urows + w * ppw * CHIP_PAIR;
    if (TRACK)
      for (int r = 0; r < rows; r++) yielded[r * 32 + lane] = 0;
    for (int r = 0; r < rows; r++) {
      const double2 u = load_u(jA + r);
      for (int par = 0; par < 2; par++)
        reinterpret_cast<double2*>(own + chip_pair_off(r >> 1, npairs, par))[32 * (r & 1) + lane] = u;
    }
    for (int q = w; q < 4; q += nw) {  // both copies: cells outside the arrays are never polled
      const double2 u = load_u(q < 2 ? y0 - 2 + q : y0 + H + q - 2);
      for (int par = 0; par < 2; par++)
        reinterpret_cast<double2*>((q < 2 ? halo_b : halo_t) + par * CHIP_PAIR)[32 * (q & 1) + lane] = u;
    }

    // what this lane polls: cell of the records (0xffffffff: none), destination in shared
    // memory (bit 0: a double-buffered row)
    const int cells = 4 * H + 4 * STREAM_COLS;
    {
      uint2* pl = polls + w * npoll * 32 + lane;
      auto cta_of = [&](int dx, int dy) { return (cy + dy) * ncx + cx + dx; };
      for (int t = 0; t < ncol; t++) {  // the columns beside the warp's rows
        const int c = t * 32 + lane, r = c >> 2, q = c & 3;
        const int col = q < 2 ? q : 28 + q;  // lanes 0, 1, 30, 31
        const int ci = x0 - 2 + col, cj = jA + r;
        uint2 e = make_uint2(0xffffffffu, 0);
        if (r < rows && ci >= 0 && ci < nx && cj < ny) {
          e.x = cta_of(q < 2 ? -1 : 1, 0) * cells + (w * rows + r) * 4 + (q < 2 ? 2 + q : q - 2);
          const int pq = r >> 1;
          e.y = (uint32_t)(own - urows) + chip_pair_off(pq, npairs, 0) + ((r & 1) * 32 + col) * 16;
          if (pq == 0 || pq == npairs - 1) e.y |= 1;
        }
        pl[t * 32] = e;
      }
      for (int t = ncol; t < npoll; t++) {  // the two rows below and above the tile
        const int q = (t - ncol) * nw + w;     // row below: 0, 1; above: 2, 3
        const bool below = q < 2;
        const int r = q & 1, cj = below ? y0 - 2 + r : y0 + H + r;
        uint2 e = make_uint2(0xffffffffu, 0);
        if (q < 4 && i >= 0 && i < nx && cj >= 0 && cj < ny) {
          const int dy = below ? -1 : 1, row = below ? H - 2 + r : r;
          if (lane < 2) e.x = cta_of(-1, dy) * cells + row * 4 + 2 + lane;
          else if (lane >= 30) e.x = cta_of(1, dy) * cells + row * 4 + lane - 30;
          else e.x = cta_of(0, dy) * cells + 4 * H + (below ? 2 * STREAM_COLS : 0) + r * STREAM_COLS + lane - 2;
          e.y = ((uint32_t)((below ? halo_b : halo_t) - urows) + (r * 32 + lane) * 16) | 1;
        }
        pl[t * 32] = e;
      }
    }
    group_barrier_or(1 + group, 32 * nw, 0);

    // V of the warp's rows to tensor memory (a warp reaches 32 of its 128 lanes)
    constexpr int VW = sizeof(VPair<TV>) / 4;
    const uint32_t vmem = s_tmem + ((uint32_t)(32 * (wc & 3)) << 16) + (uint32_t)((wc >> 2) * npairs * VW);
    TV* __restrict__ fvx = static_cast<TV*>(f.vx);
    TV* __restrict__ fvy = static_cast<TV*>(f.vy);
    const bool col_own = lane >= 2 && lane < 2 + STREAM_COLS && i < nx;
    for (int q = 0; q < npairs; q++) {
      VPair<TV> v;
      for (int r = 0; r < 2; r++) {
        const int j = jA + 2 * q + r;
        const bool in = col_own && j < ny;
        v.set(2 * r, in ? fvx[j * pitch + i] : (TV)0);
        v.set(2 * r + 1, in ? fvy[j * pitch + i] : (TV)0);
      }
      tmem_st(vmem + q * VW, v.w);
    }
    tmem_st_wait();

    const char* rd_below = w > 0 ? own - ppw * CHIP_PAIR + (npairs == 1 ? 0 : 2 * CHIP_PAIR) : halo_b;
    const char* rd_above = w < nw - 1 ? own + ppw * CHIP_PAIR : halo_t;
    const bool interior = x0 - 2 >= 1 && x0 + 29 <= nx - 3 && jA >= 3 && jA + rows <= ny - 2;
    const size_t rim_parity = (size_t)(ncx * ncy) * cells * RIM_BYTES;
    int it = 0;
    for (;; it++) {
      const int par = it & 1;
      if (jA < ny) {
        const char* below = rd_below + par * CHIP_PAIR;
        const char* above = rd_above + par * CHIP_PAIR;
        const uint8_t* ix = idx + (w * rows) * 32;
        auto march = [&](auto plastic_c) {
          constexpr bool P = decltype(plastic_c)::value;
          auto rows_of = [&](auto np_c) {
            constexpr int NP = decltype(np_c)::value;
            if (interior)
              chip_march<P, false, NP, TV, TRACK>(g, mats, ix, below, own, above, npairs, par, i, jA, vmem, yielded);
            else
              chip_march<P, true, NP, TV, TRACK>(g, mats, ix, below, own, above, npairs, par, i, jA, vmem, yielded);
          };
          if (npairs == 1) rows_of(std::integral_constant<int, 1>{});
          else if (npairs == 2) rows_of(std::integral_constant<int, 2>{});
          else if (npairs == 3) rows_of(std::integral_constant<int, 3>{});
          else rows_of(std::integral_constant<int, 0>{});
        };
        if (PLASTIC == 1 || (PLASTIC == 2 && job.plastic)) march(std::true_type{});
        else march(std::false_type{});
      }
      if (it + 1 >= n_iter) break;
      __syncwarp();
      const uint32_t tag = (uint32_t)it + 1;  // the records start as zeros
      char* out = job.rim + par * rim_parity + (size_t)tile * cells * RIM_BYTES;
      const char* in = job.rim + par * rim_parity;
      auto put = [&](int cell, int r, int col) {
        rim_put(out + cell * RIM_BYTES,
                reinterpret_cast<const double2*>(own + chip_pair_off(r >> 1, npairs, par ^ 1))[(r & 1) * 32 + col], tag);
      };
      if (jA < ny) {
        for (int c = lane; c < 4 * rows; c += 32) put(w * rows * 4 + c, c >> 2, (c & 3) < 2 ? 2 + (c & 3) : 26 + (c & 3));
        if (w == 0 && cy > 0)
          for (int r = 0; r < 2; r++)
            if (lane < STREAM_COLS) put(4 * H + r * STREAM_COLS + lane, r, 2 + lane);
        if (w == nw - 1 && cy < ncy - 1)
          for (int r = 0; r < 2; r++)
            if (lane < STREAM_COLS) put(4 * H + (2 + r) * STREAM_COLS + lane, rows - 2 + r, 2 + lane);
      }
      int failed = 0;
      for (int t0 = 0; t0 < npoll && !failed; t0 += kRimInFlight) {
        uint2 e[kRimInFlight];
        RimRecord rec[kRimInFlight];
        bool wait[kRimInFlight];
#pragma unroll
        for (int k = 0; k < kRimInFlight; k++) {
          e[k].x = 0xffffffffu;
          if (t0 + k < npoll) e[k] = polls[(w * npoll + t0 + k) * 32 + lane];
          wait[k] = e[k].x != 0xffffffffu;
        }
        unsigned tries = 0;
        unsigned long long since = 0;
        for (;;) {
          bool any = false;
#pragma unroll
          for (int k = 0; k < kRimInFlight; k++)
            if (wait[k]) rim_get(in + (size_t)e[k].x * RIM_BYTES, rec[k]);
#pragma unroll
          for (int k = 0; k < kRimInFlight; k++) {
            if (wait[k]) wait[k] = !rec[k].ready(tag);
            any |= wait[k];
          }
          if (!__any_sync(0xffffffffu, any)) break;
          if ((++tries & 1023u) == 0) {  // bounded: look at the clock and the error flag now and then
            const unsigned long long now = global_ns();
            if (since == 0) since = now;
            if (now - since > a.timeout_ns) atomicExch(job.flag, 1u);
            if (__any_sync(0xffffffffu, *reinterpret_cast<volatile unsigned*>(job.flag) != 0)) {
              failed = 1;
              break;
            }
          }
        }
#pragma unroll
        for (int k = 0; k < kRimInFlight; k++) {
          if (e[k].x == 0xffffffffu) continue;
          const uint32_t off = (e[k].y & ~1u) + ((e[k].y & 1u) ? (uint32_t)(par ^ 1) * CHIP_PAIR : 0u);
          *reinterpret_cast<double2*>(urows + off) = rec[k].value();
        }
      }
      if (group_barrier_or(1 + group, 32 * nw, failed)) break;
    }

    // back to global memory: U of the last copy written, V
    if (jA < ny) {
      __syncwarp();
      double* uxo = f.ux[src ^ (n_iter & 1)];
      double* uyo = f.uy[src ^ (n_iter & 1)];
      const int par = (it & 1) ^ 1;
      for (int q = 0; q < npairs; q++) {
        VPair<TV> v;
        tmem_ld(vmem + q * VW, v.w);
        tmem_ld_wait(v.w);
        for (int r = 0; r < 2; r++) {
          const int j = jA + 2 * q + r;
          if (col_own && j < ny) {
            const double2 u = reinterpret_cast<const double2*>(own + chip_pair_off(q, npairs, par))[32 * r + lane];
            uxo[j * pitch + i] = u.x;
            uyo[j * pitch + i] = u.y;
            fvx[j * pitch + i] = v.get(2 * r);
            fvy[j * pitch + i] = v.get(2 * r + 1);
            if (TRACK) const_cast<uint8_t*>(f.mask)[j * pitch + i] |= yielded[(2 * q + r) * 32 + lane];
          }
        }
      }
    }
  }
  __syncthreads();
  if (wc == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(s_tmem));
}

}  // namespace ep2d
