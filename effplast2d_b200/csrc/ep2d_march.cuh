// ep2d_march.cuh -- the march of one warp up the rows of a strip, two rows per step: the
// iteration ComputeStress -> ComputeJ2 -> ComputePlasticity -> ComputeDisp
// (EffPlast2D.cu:3-177) of 28 owned columns (lanes 2..29; lanes 0, 1, 30, 31 are halo) and
// 2 npairs rows, shared by the on-chip form (ep2d_iter_chip.cuh) and the stream form
// (ep2d_iter_stream.cuh), which differ in where the rows come from and go to.
//
// Step p takes U of rows ka = jA - 2 + 2p and ka + 1, forms the trial stresses of rows
// ka - 1 and ka, returns rows ka - 2 and ka - 1 and updates the faces of those two rows (own
// pair p - 2).  Neighbouring columns come from warp shuffles.  Two rows per step halve what a
// step costs besides its arithmetic and give the scheduler two independent chains; the carried
// values (the last row's U, trials and pair sums, the returned row below) need no
// register moves but once per two rows.
//
// The radial return is skipped where no lane of the warp yields in either row (a warp vote):
// the four factors, each a reciprocal square root, are a third of a step's instructions, and
// most warps of a solve are elastic outside the plastic zones.  Inside, every lane
// evaluates the factor of a value that is in range (its own J2^2, or the limit) and
// selects, so there is no branch around each square root.
//
// Nodes and corners outside the grid have zero material constants (like those in a pore),
// so their stresses are 0 whatever U is there; only the clamped 2x2 corner block of the node
// return and the faces on the boundary differ at the edges (EDGE).
#pragma once

#include <type_traits>

#include "ep2d_stencil.cuh"
#include "ep2d_types.hpp"

namespace ep2d {

template <typename T>
struct Vec2T;
template <>
struct Vec2T<double> {
  using type = double2;
};
template <>
struct Vec2T<float> {
  using type = float2;
};
template <typename T>
using Vec2 = typename Vec2T<T>::type;

// material constants of a node (K, 2G) and of the corner of the same indices (a quarter of the four
// nodes' G); by the 7-bit index (node's M_MAT | M_NODE) | corner_index << 2
template <typename T>
struct __align__(16) MatT {
  T k, g2, g4, pad;
};
constexpr int N_MATS = 128;

// c = corner table index of the corner (i, j) from the mask bytes of nodes (i, j) and
// (i, j + 1); the four material bits of g4z's index: bit 0 node (i, j), bit 3 (i+1, j),
// bit 1 (i, j+1), bit 4 (i+1, j+1); bit 2 the corner's pore bit
__device__ __forceinline__ int corner_index(int m_j, int m_j1) {
  return (m_j & (M_MAT | M_CORNER | M_MAT_R)) | ((m_j1 & (M_MAT | M_MAT_R)) << 1);
}
__device__ __forceinline__ double g4z_entry(int c, double G0, double Gp) {
  return (c & 4) ? 0.0 : corner_g4(c & 1, (c >> 3) & 1, (c >> 1) & 1, (c >> 4) & 1, G0, Gp);
}
template <typename T>
__device__ __forceinline__ MatT<T> mat_entry(const Geo& g, int t) {
  MatT<T> m{(T)0, (T)0, (T)g4z_entry(t >> 2, g.G0, g.Gp), (T)0};
  if (!(t & M_NODE)) {
    m.k = (T)((t & M_MAT) ? g.Kp : g.K0);
    m.g2 = (T)__dmul_rn(2.0, (t & M_MAT) ? g.Gp : g.G0);
  }
  return m;
}

// The displacement arrays of a form: FP64 U, or the FP32 bulk's perturbations u'.
template <typename TU>
__device__ __forceinline__ TU* u_field(const Fields& f, bool y, int buf);
template <>
__device__ __forceinline__ double* u_field<double>(const Fields& f, bool y, int buf) {
  return y ? f.uy[buf] : f.ux[buf];
}
template <>
__device__ __forceinline__ float* u_field<float>(const Fields& f, bool y, int buf) {
  return y ? f.uy32[buf] : f.ux32[buf];
}

template <typename T>
__device__ __forceinline__ T shfl_idx(T v, int src) { return __shfl_sync(0xffffffffu, v, src); }
template <typename T>
__device__ __forceinline__ T shfl_dn(T v) { return __shfl_down_sync(0xffffffffu, v, 1); }
template <typename T>
__device__ __forceinline__ T shfl_up1(T v) { return __shfl_up_sync(0xffffffffu, v, 1); }

__device__ __forceinline__ double rsqrt_of(double x) { return rsqrt(x); }
__device__ __forceinline__ float rsqrt_of(float x) { return rsqrtf(x); }

// Io, the rows' source and destination:
//   SELECT                          how the node sums at the grid's lowest and highest rows are formed
//   begin<STAGE>(p)                 before step p's rows are read
//   rows(p, ua, uar, ub, ubr)       (Ux, Uy) of rows ka and ka + 1, this column's and the next one's
//   mat(p, r)                       materials of row ka - 1 (r = 0) or ka (r = 1)
//   old(p, u0, u1, v)               U and V = {vx, vy of the lower row, of the upper} of own pair p - 2
//   store(p, u0, u1, v)             their new values
//   yields(p, n0, n1, c0, c1)       TRACK: own pair p - 2's nodes and corners that yield
// DOWN: the rows are counted from the top: row j here is row ny - 1 - j of the nodes, Ux and Vx, row
// ny - j of Uy and Vy, corner row ny - 2 - j.  Differences along y then have their operands in the
// other order, and every value is formed from the same operands as in the march up.
// T: arithmetic and displacement type, TV: velocity storage.  T = float: the FP32 bulk's
// perturbations about the affine field.
template <typename T, typename TV, bool PLASTIC, bool EDGE, int NP, bool TRACK, int UNROLL, bool DOWN = false,
          typename Io>
__device__ __forceinline__ void pair_march(const Geo& g, Io& io, int npairs_in, int i, int jA) {
  using U2 = Vec2<T>;
  const int npairs = NP ? NP : npairs_in;
  const int lane = threadIdx.x & 31;
  const int nx = g.nx, ny = g.ny;
  const T rdX = (T)g.rdX, rdY = (T)g.rdY, third = (T)(1.0 / 3.0);
  const T coh = (T)g.coh, coh2 = (T)g.coh2, coh4 = (T)g.coh4, coh2x16 = (T)g.coh2x16;
  const T dT = (T)g.dT, cX = (T)g.cX, cY = (T)g.cY, dtrX = (T)g.dtrX, dtrY = (T)g.dtrY;
  const T exx0 = (T)g.exx0, eyy0 = (T)g.eyy0, exy0 = (T)g.exy0;  // FP32 bulk only
  int sa = 0, sb = 0;  // lanes of the node's clamped corner columns
  if (EDGE) {
    const int a = min(max(i - 1, 0), nx - 3) - i;
    sa = min(max(lane + a, 0), 31);
    sb = min(max(lane + a + 1, 0), 31);
  }

  T uxc = 0, uxc_r = 0, uyc = 0;    // U of the last row read
  T pb = 0, xb = 0, yb = 0, cb = 0; // trial stresses of the last row
  T hz = 0, h0 = 0, h1 = 0;         // corner pair sums of the last three rows
  T syq = 0, cq = 0, cq_l = 0;      // returned: total syy, corner of the row below

  auto diff_y = [](T upper, T lower) { return DOWN ? sub_rn(lower, upper) : sub_rn(upper, lower); };
  auto trial = [&](const MatT<T>& m, T ux, T ux_r, T uy, T ux1_r, T uy1, T uy1_r, T& p, T& x, T& y, T& c) {
    if constexpr (std::is_same<T, float>::value) {
      node_trial(sub_rn(ux_r, ux), diff_y(uy1, uy), exx0, eyy0, m.k, m.g2, rdX, rdY, third, p, x, y);
      c = corner_trial(m.g4, diff_y(ux1_r, ux_r), sub_rn(uy1_r, uy1), exy0, rdX, rdY);
    } else {
      node_trial(sub_rn(ux_r, ux), diff_y(uy1, uy), m.k, m.g2, rdX, rdY, third, p, x, y);
      c = corner_trial(m.g4, diff_y(ux1_r, ux_r), sub_rn(uy1_r, uy1), rdX, rdY);
    }
  };
  auto corner_pair = [&](T c) {
    return EDGE ? add_rn(shfl_idx(c, sa), shfl_idx(c, sb)) : add_rn(shfl_up1(c), c);
  };
  // The 4-corner sum of node row j adds the pair sums of corner rows j - 1 and j; of row 0 those of
  // rows 0 and 1, of row ny - 1 those of rows ny - 3 and ny - 2 (EDGE).  So pair row ny - 1 takes row
  // ny - 3's place, and row -1 that of row 1: one select on a pair sum instead of three sums to select
  // from (Io::SELECT).
  constexpr bool SELECT = Io::SELECT;
  auto pair_above = [&](int row, T h, T h2) { return SELECT && EDGE && row == ny - 1 ? h2 : h; };
  auto corner_sum = [&](int j, bool first, T hm2, T hm1, T hj, T hp1) {  // pair sums of rows j - 2 .. j + 1
    if (EDGE && !SELECT) return j == 0 ? add_rn(hj, hp1) : j == ny - 1 ? add_rn(hm2, hm1) : add_rn(hm1, hj);
    return add_rn(EDGE && first && j == 0 ? hp1 : hm1, hj);
  };
  // 16 J2^2 of a corner of row j from the node deviators of rows j and j + 1
  auto corner_j2 = [&](T x, T y, T c, T xn, T yn) {
    const T vx = add_rn(x, xn), vy = add_rn(y, yn);
    const T tx = add_rn(vx, shfl_dn(vx)), ty = add_rn(vy, shfl_dn(vy));
    return corner_j2sq16(tx, ty, c);
  };
  auto factor = [&](T j2, T lim2, T lim) {  // return_factor
    const bool yields = j2 > lim2;
    const T r = mul_rn(lim, rsqrt_of(yields ? j2 : lim2));
    return yields ? r : (T)1;
  };
  // faces of row j: new velocities and displacements from the old ones
  auto face = [&](int j, T sx, T sx_l, T sy, T cw_l, TV& vx, TV& vy, U2& u) {
    const T vxo = (T)vx, vyo = (T)vy;
    const TV vxs = (TV)face_velocity_s(vxo, cX, sub_rn(sx, sx_l), dtrX, diff_y(cw_l, cq_l), dtrY);
    const TV vys = (TV)face_velocity_s(vyo, cY, diff_y(sy, syq), dtrY, sub_rn(cq, cq_l), dtrX);
    if (EDGE) {  // a face the reference leaves alone keeps its velocity
      if (i > 0 && j > 0 && j < ny - 1) vx = vxs;
      if (i > 0 && i < nx - 1 && j > 0) vy = vys;
    } else {
      vx = vxs;
      vy = vys;
    }
    u.x = advance(u.x, (T)vx, dT);  // the displacement moves by the stored velocity
    u.y = advance(u.y, (T)vy, dT);
  };

  auto pair = [&](auto stage_c, int p) {
    constexpr int STAGE = decltype(stage_c)::value;  // 0: trial of row ka, 1: and the return of ka - 1, 2: all
    io.template begin<STAGE>(p);
    U2 ua, uar, ub, ubr;
    io.rows(p, ua, uar, ub, ubr);
    T p1 = 0, x1 = 0, y1 = 0, c1 = 0, p2, x2, y2, c2, hs1 = 0, hs2 = 0;
    if constexpr (STAGE >= 1) {
      trial(io.mat(p, 0), uxc, uxc_r, uyc, uar.x, ua.y, uar.y, p1, x1, y1, c1);
      if (PLASTIC) hs1 = pair_above(jA + 2 * p - 3, corner_pair(c1), h0);
    }
    trial(io.mat(p, 1), ua.x, uar.x, ua.y, ubr.x, ub.y, ubr.y, p2, x2, y2, c2);
    if (PLASTIC) hs2 = pair_above(jA + 2 * p - 2, corner_pair(c2), h1);
    const int ja = jA + 2 * p - 4;  // row ka - 2
    if constexpr (STAGE == 2) {
      T xr0 = xb, yr0 = yb, cw0 = cb, xr1 = x1, yr1 = y1, cw1 = c1;
      if (PLASTIC) {
        const T n0 = node_j2sq_h(xb, yb, corner_sum(ja, true, hz, h0, h1, hs1));
        const T n1 = node_j2sq_h(x1, y1, corner_sum(ja + 1, false, h0, h1, hs1, hs2));
        const T m0 = corner_j2(xb, yb, cb, x1, y1), m1 = corner_j2(x1, y1, c1, x2, y2);
        if (__any_sync(0xffffffffu, n0 > coh2 || n1 > coh2 || m0 > coh2x16 || m1 > coh2x16)) {
          const T f0 = factor(n0, coh2, coh), f1 = factor(n1, coh2, coh);
          xr0 = mul_rn(xb, f0);
          yr0 = mul_rn(yb, f0);
          cw0 = mul_rn(cb, factor(m0, coh2x16, coh4));
          xr1 = mul_rn(x1, f1);
          yr1 = mul_rn(y1, f1);
          cw1 = mul_rn(c1, factor(m1, coh2x16, coh4));
          if (TRACK) {  // J2 > coh from the trial stresses (get_sigma_2D.m:126-138); corners inside the grid
            const bool c_in = !EDGE || i < nx - 1;
            io.yields(p, n0 > coh2, n1 > coh2, c_in && (!EDGE || ja < ny - 1) && m0 > coh2x16,
                      c_in && (!EDGE || ja + 1 < ny - 1) && m1 > coh2x16);
          }
        }
      }
      const T sx0 = sub_rn(xr0, pb), sy0 = sub_rn(yr0, pb), sx1 = sub_rn(xr1, p1), sy1 = sub_rn(yr1, p1);
      const T cw0_l = shfl_up1(cw0), sx0_l = shfl_up1(sx0);
      const T cw1_l = shfl_up1(cw1), sx1_l = shfl_up1(sx1);
      U2 u0, u1;
      TV v[4];
      io.old(p, u0, u1, v);
      face(ja, sx0, sx0_l, sy0, cw0_l, v[0], v[1], u0);
      syq = sy0;
      cq = cw0;
      cq_l = cw0_l;
      face(ja + 1, sx1, sx1_l, sy1, cw1_l, v[2], v[3], u1);
      syq = sy1;
      cq = cw1;
      cq_l = cw1_l;
      io.store(p, u0, u1, v);
    } else if constexpr (STAGE == 1) {
      T yr = y1;
      cq = c1;
      if (PLASTIC) {
        yr = mul_rn(y1, factor(node_j2sq_h(x1, y1, corner_sum(ja + 1, false, h0, h1, hs1, hs2)), coh2, coh));
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
  };
  pair(std::integral_constant<int, 0>{}, 0);
  pair(std::integral_constant<int, 1>{}, 1);
#pragma unroll (NP ? NP : UNROLL)
  for (int p = 2; p <= npairs + 1; p++) pair(std::integral_constant<int, 2>{}, p);
}

}  // namespace ep2d
