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
// fence, flag or grid-wide barrier (each 64-bit {word, tag} is an element of one vector
// store and valid on its own).  Records are double-buffered by iteration parity: a CTA
// overwrites iteration t's records in iteration t + 2, after it has read its neighbours'
// records of t + 1, which they wrote after reading all of t's.  Waits are bounded.  Each CTA counts
// itself in the RVE's state word as it starts; where one cannot (other work holds its SM),
// its neighbours' waits give up after start_ns, every CTA leaves without having written the
// state, and the host runs the iterations in another form.  A wait for a CTA that has started
// gives up after records_ns, and the host reports the RVE as failed.
//
// Within a CTA the two lowest and two highest rows of a warp are read by the warps below
// and above and are double-buffered by parity; the rows between are updated in place.
// One barrier of the tile's warps per iteration.  All CTAs must be resident at once
// (cooperative launch, one CTA per SM).
//
// What bounds it: on grids up to ~400^2 latency, the rim exchange (1.4 us of an iteration
// with the march left out) and one warp's march; on larger ones the issue of the march's
// instructions (1024^2: 198 warp instructions per strip row, issued in 63 % of the cycles).  Measured, us per iteration, the form the library took before / this one
// (FP64): elastic 128^2 4.2 / 1.51, 1024^2 15.5 / 5.9; with the return map 128^2 5.8 / 2.05, 256^2
// 6.2 / 2.50, 512^2 8.9 / 3.75, 768^2 14.3 / 6.83, 1024^2 16.3 / 9.96.
#pragma once

#include "ep2d_march.cuh"
#include "ep2d_types.hpp"

namespace ep2d {

// row pairs per turn of the march's loop: 2 measured best (1024^2, 16 rows: 9.85 us an
// iteration; 1: 10.5, 4: 9.94 with spills)
constexpr int kChipUnroll = 2;

// shared memory, in bytes, u = the size of a displacement: materials, U rows (32 columns of
// (Ux, Uy)) in pairs, the material index of every (row, column), and the poll list
__host__ __device__ constexpr int chip_pair_bytes(int u) { return 2 * 32 * 2 * u; }
__host__ __device__ constexpr int chip_pairs_per_warp(int rows) { return rows == 2 ? 2 : rows / 2 + 2; }
// cells a lane polls: of the columns beside its warp's rows (4 per row), of the rows below
// and above the tile (2 x 2 x 32 cells, spread over the group's warps)
__host__ __device__ constexpr int chip_col_polls(int rows) { return (4 * rows + 31) / 32; }
__host__ __device__ constexpr int chip_polls(int warps, int rows) {
  return chip_col_polls(rows) + (4 + warps - 1) / warps;
}
__host__ __device__ constexpr size_t chip_group_bytes(int warps, int rows, int u) {
  return (size_t)(warps * chip_pairs_per_warp(rows) + 4) * chip_pair_bytes(u) + (size_t)(warps * rows + 4) * 32 +
         (size_t)warps * chip_polls(warps, rows) * 32 * sizeof(uint2);
}
// with tracking, a byte of yield bits per (row, column) behind the groups' regions
__host__ __device__ constexpr size_t chip_smem_bytes(int groups, int warps, int rows, bool track = false, int u = 8) {
  return N_MATS * 4 * u + groups * (chip_group_bytes(warps, rows, u) + (track ? warps * rows * 32 : 0));
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

// The time a wait has taken in ns, looked at now and then: time between two looks counts as at most
// 10 ms, so that time in which the GPU runs another context does not.
struct ChipClock {
  unsigned waited = 0, last = 0;  // in units of 1024 ns
  __device__ __forceinline__ unsigned long long look() {
    const unsigned now = (unsigned)(global_ns() >> 10) | 1u;
    if (last) waited += min(now - last, 9766u);
    last = now;
    return (unsigned long long)waited << 10;
  }
};
// A look at the job's state word by a warp that has waited this long: gives up where its limit has passed
// (the mark shows at the next look); true if the launch has failed.
__device__ __forceinline__ bool chip_look(const ChipJob& job, unsigned long long waited, unsigned long long start_ns,
                                          unsigned long long records_ns) {
  const unsigned w = *reinterpret_cast<volatile unsigned*>(job.state);
  const bool all = (w & CHIP_COUNT) == job.full;
  if (waited > (all ? records_ns : start_ns))
    atomicCAS(job.state, w, w | (all ? CHIP_STALLED : CHIP_GAVE_UP));
  return __any_sync(0xffffffffu, (w & CHIP_FAILED) != 0);
}
// Gives up waiting for a CTA that has not started, unless it just has.
__device__ __forceinline__ void chip_give_up(const ChipJob& job) {
  unsigned w = *reinterpret_cast<volatile unsigned*>(job.state);
  while (!(w & CHIP_FAILED)) {
    if ((w & CHIP_COUNT) == job.full) return;
    const unsigned old = atomicCAS(job.state, w, w | CHIP_GAVE_UP);
    if (old == w) return;
    w = old;
  }
}
// Waits until all CTAs of the job have started; false if the launch has failed.
__device__ __forceinline__ bool chip_all_started(const ChipJob& job, unsigned long long start_ns) {
  ChipClock clock;
  for (unsigned tries = 1;; tries++) {
    const unsigned w = *reinterpret_cast<volatile unsigned*>(job.state);
    if (__any_sync(0xffffffffu, (w & CHIP_FAILED) != 0)) return false;
    if (__all_sync(0xffffffffu, (w & CHIP_COUNT) == job.full)) return true;
    if ((tries & 1023u) == 0 && clock.look() > start_ns) chip_give_up(job);
  }
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
// Record of a cell: {lo, tag, hi, tag} of Ux and of Uy, one 256-bit access; for float
// displacements {Ux, tag, Uy, tag}, one 128-bit access.  The accesses' elements are the 64-bit
// {word, tag}, so no element shows a tag without its word; they are taken apart inside the
// statement (packed with shifts outside it 1024^2 took 3 % longer).
template <typename T>
struct RimRecord;
template <>
struct RimRecord<double> {
  static constexpr int BYTES = 32;
  uint32_t w[8];
  __device__ bool ready(uint32_t tag) const { return ((w[1] ^ tag) | (w[3] ^ tag) | (w[5] ^ tag) | (w[7] ^ tag)) == 0; }
  __device__ double2 value() const {
    return make_double2(__hiloint2double((int)w[2], (int)w[0]), __hiloint2double((int)w[6], (int)w[4]));
  }
  __device__ void get(const char* rec) {
    asm volatile(
        "{\n .reg .b64 a, b, c, d;\n ld.relaxed.gpu.global.v4.b64 {a,b,c,d}, [%8];\n mov.b64 {%0,%1}, a;\n"
        " mov.b64 {%2,%3}, b;\n mov.b64 {%4,%5}, c;\n mov.b64 {%6,%7}, d;\n}"
                 : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7])
                 : "l"(rec)
                 : "memory");
  }
  static __device__ void put(char* rec, const double2& u, uint32_t tag) {
    asm volatile(
        "{\n .reg .b64 a, b, c, d;\n mov.b64 a, {%1,%5};\n mov.b64 b, {%2,%5};\n mov.b64 c, {%3,%5};\n"
        " mov.b64 d, {%4,%5};\n st.relaxed.gpu.global.v4.b64 [%0], {a,b,c,d};\n}" ::"l"(rec),
        "r"(__double2loint(u.x)), "r"(__double2hiint(u.x)), "r"(__double2loint(u.y)), "r"(__double2hiint(u.y)), "r"(tag)
        : "memory");
  }
};
template <>
struct RimRecord<float> {
  static constexpr int BYTES = 16;
  uint32_t w[4];
  __device__ bool ready(uint32_t tag) const { return ((w[1] ^ tag) | (w[3] ^ tag)) == 0; }
  __device__ float2 value() const { return make_float2(__uint_as_float(w[0]), __uint_as_float(w[2])); }
  __device__ void get(const char* rec) {
    asm volatile(
        "{\n .reg .b64 a, b;\n ld.relaxed.gpu.global.v2.b64 {a,b}, [%4];\n mov.b64 {%0,%1}, a;\n mov.b64 {%2,%3}, b;\n}"
                 : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3])
                 : "l"(rec)
                 : "memory");
  }
  static __device__ void put(char* rec, const float2& u, uint32_t tag) {
    asm volatile(
        "{\n .reg .b64 a, b;\n mov.b64 a, {%1,%3};\n mov.b64 b, {%2,%3};\n st.relaxed.gpu.global.v2.b64 [%0], {a,b};\n}" ::
            "l"(rec),
        "r"(__float_as_uint(u.x)), "r"(__float_as_uint(u.y)), "r"(tag)
        : "memory");
  }
};
// where a warp's row pairs lie: pair q of its rows/2, copy `par` of the double-buffered ones
template <typename T>
__device__ __forceinline__ uint32_t chip_pair_off(int q, int npairs, int par) {
  constexpr uint32_t PAIR = chip_pair_bytes(sizeof(T));
  if (q == 0) return par * PAIR;
  if (q == npairs - 1) return (2 + par) * PAIR;
  return (3 + q) * PAIR;
}

// Rows of one warp's tile part for pair_march: U in shared memory (from copy `par` to copy
// par ^ 1), V in tensor memory.  NP: the number of row pairs where it is known (1 to 3: the march
// unrolled, so that its rows' chains overlap: 256^2, 2 rows, 2.70 -> 2.54 us an iteration; 448^2,
// 4 rows, 3.76 -> 3.55; 512^2, 6 rows, 4.29 -> 4.07), else 0.
// SEL: SELECT of the march.  The warps at the grid's edges set the pace of all, and with it their rows take
// fewer sums (us per iteration: 128^2 2.13 -> 2.04, 256^2 2.54 -> 2.48, 512^2 3.91 -> 3.73, 601^2 4.49 ->
// 4.36, FP32 768^2 4.60 -> 4.35).  The FP64 kernels with three records in flight have no register to
// spare for it (768^2 6.81 -> 7.13, 1024^2 9.98 -> 10.59).
template <typename T, typename TV, bool EDGE, int NP, bool SEL>
struct ChipIo {
  using U2 = Vec2<T>;
  static constexpr bool SELECT = SEL;
  static constexpr int VW = sizeof(VPair<TV>) / 4;
  const MatT<T>* mats;
  const uint8_t* idx;       // material indices of row jA - 2 on, 32 per row, this lane's column
  const char *below, *above;  // the row pairs below and above the warp's own
  char* own;
  const char* rd;           // the pair read at this step, and at the one before
  const char* rd_prev;
  int npairs, par, right, rows_left;  // rows_left: own rows inside the grid (EDGE)
  bool col_own;
  uint32_t vmem;
  uint8_t* yielded;         // TRACK: yield bits of the warp's rows, this lane's column
  VPair<TV> v;

  template <int STAGE>
  __device__ __forceinline__ void begin(int p) {
    // the other lanes have read the rows this step overwrites (with one or two pairs every
    // row is double-buffered)
    if (NP == 0 || NP > 2) __syncwarp();
    if constexpr (STAGE == 2) tmem_ld(vmem + (p - 2) * VW, v.w);
    rd_prev = rd;
    rd = p == 0 ? below : p <= npairs ? own + chip_pair_off<T>(p - 1, npairs, par) : above;
  }
  __device__ __forceinline__ void rows(int, U2& ua, U2& uar, U2& ub, U2& ubr) {
    const U2* r = reinterpret_cast<const U2*>(rd) + (threadIdx.x & 31);
    ua = r[0];
    uar = r[right];
    ub = r[32];
    ubr = r[32 + right];
  }
  __device__ __forceinline__ const MatT<T>& mat(int p, int r) { return mats[idx[(2 * p - 1 + r) * 32]]; }
  __device__ __forceinline__ void old(int, U2& u0, U2& u1, TV (&vv)[4]) {
    const U2* r = reinterpret_cast<const U2*>(rd_prev) + (threadIdx.x & 31);
    u0 = r[0];
    u1 = r[32];
    tmem_ld_wait(v.w);
#pragma unroll
    for (int k = 0; k < 4; k++) vv[k] = v.get(k);
  }
  __device__ __forceinline__ void store(int p, const U2& u0, const U2& u1, const TV (&vv)[4]) {
#pragma unroll
    for (int k = 0; k < 4; k++) v.set(k, vv[k]);
    tmem_st(vmem + (p - 2) * VW, v.w);
    U2* un = reinterpret_cast<U2*>(own + chip_pair_off<T>(p - 2, npairs, par ^ 1)) + (threadIdx.x & 31);
    if (col_own && (!EDGE || 2 * p - 4 < rows_left)) un[0] = u0;
    if (col_own && (!EDGE || 2 * p - 3 < rows_left)) un[32] = u1;
  }
  __device__ __forceinline__ void yields(int p, bool n0, bool n1, bool c0, bool c1) {
    uint8_t* y = yielded + 2 * (p - 2) * 32;
    y[0] |= (n0 ? M_YN : 0) | (c0 ? M_YC : 0);
    y[32] |= (n1 ? M_YN : 0) | (c1 ? M_YC : 0);
  }
};

// a.n_iter plain iterations of every job's RVE from its buffer `src`, ending in buffer
// src ^ (n_iter & 1) (n_iter >= 2: when the buffers coincide, a tile is written back only after
// its neighbours have read it).  CTAs of groups of a.warps warps, a group per tile, a.rows rows per
// warp.  rim: records [2][tile][4 H + 112 cells].  PLASTIC 0, 1: all jobs; 2: per job.
// TRACK: also mark the nodes and corners that yield at any of the iterations (M_YN, M_YC).
// WARPS: the most warps of a CTA.  A shape of 8 or 12 warps per SM leaves the march 255 or 168
// registers instead of 128, and the unrolled rows overlap better (us per iteration: 128^2
// elastic 1.63 -> 1.50, NL=3 2.28 -> 2.10 with 4 warps; 256^2 2.66 -> 2.56, 512^2 elastic 2.40 ->
// 2.29, NL=3 4.10 -> 3.96 with 10 and 12).
// FLY: records a lane has in flight while it polls.  Tiles of 10 rows per warp and more have
// three per lane; in one go they cost one round trip (1024^2 10.08 -> 9.93 us an iteration; elastic RVEs
// gain nothing: 5.82, 5.91).  Where
// two do, a third costs 2 %, and a fourth spills the march.
template <int PLASTIC, int JOBS, typename T, typename TV, bool TRACK = false, int WARPS = CHIP_WARPS, int FLY = 3>
__global__ void __launch_bounds__(32 * WARPS, 1) k_iter_chip(const __grid_constant__ ChipArgs<JOBS> a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ uint32_t s_tmem;
  using U2 = Vec2<T>;
  constexpr int US = sizeof(T), PAIR = chip_pair_bytes(US), RIM_BYTES = RimRecord<T>::BYTES;
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
  // counted before anything is published: a tile whose neighbours' records have come knows they started
  if (__syncthreads_or(threadIdx.x == 0 && (atomicAdd(job.state, 1u) & CHIP_FAILED))) return;

  MatT<T>* mats = reinterpret_cast<MatT<T>*>(smem_raw);
  char* urows = reinterpret_cast<char*>(smem_raw) + N_MATS * sizeof(MatT<T>) + group * chip_group_bytes(nw, rows, US);
  char* halo_b = urows + nw * ppw * PAIR;
  char* halo_t = halo_b + 2 * PAIR;  // the rows below and above the tile, two copies each
  uint8_t* idx = reinterpret_cast<uint8_t*>(halo_t + 2 * PAIR);
  uint2* polls = reinterpret_cast<uint2*>(idx + (H + 4) * 32);
  uint8_t* yielded = smem_raw + chip_smem_bytes(groups, nw, rows, false, US) + wc * rows * 32;  // TRACK only

  if (wc == 0) {  // one CTA per SM takes all of the SM's tensor memory
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(
                     (uint32_t)__cvta_generic_to_shared(&s_tmem))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  // the recording launch that follows folds max|V| into the pair
  if ((int)blockIdx.x == job.cta0 && threadIdx.x < 2) f.vmax[threadIdx.x] = 0;
  for (int t = threadIdx.x; t < N_MATS; t += blockDim.x) mats[t] = mat_entry<T>(g, t);
  __syncthreads();
  // A tile that has gone through n iterations has records that go back to every tile up to n - 1 away, so
  // all have started when it writes the state back; with fewer iterations it has to look.
  if (!idle && (n_iter >= max(ncx, ncy) || chip_all_started(job, a.start_ns))) {
    const int i = x0 - 2 + lane;
    const int jA = y0 + w * rows;
#pragma unroll 4
    for (int r = w; r < H + 3; r += nw) idx[r * 32 + lane] = (uint8_t)chip_index(g, f.mask, i, y0 - 2 + r);

    // U of the tile and its halo, both copies of the double-buffered rows (faces outside the
    // arrays: 0; the face column nx of Ux and row ny of Uy never change)
    const T* __restrict__ ux = u_field<T>(f, false, src);
    const T* __restrict__ uy = u_field<T>(f, true, src);
    auto load_u = [&](int j) {
      U2 u;
      u.x = (i >= 0 && i <= nx && j >= 0 && j < ny) ? ux[j * pitch + i] : (T)0;
      u.y = (i >= 0 && i < nx && j >= 0 && j <= ny) ? uy[j * pitch + i] : (T)0;
      return u;
    };
    char* own = urows + w * ppw * PAIR;
    if (TRACK)
      for (int r = 0; r < rows; r++) yielded[r * 32 + lane] = 0;
#pragma unroll 4
    for (int r = 0; r < rows; r++) {
      const U2 u = load_u(jA + r);
      for (int par = 0; par < 2; par++)
        reinterpret_cast<U2*>(own + chip_pair_off<T>(r >> 1, npairs, par))[32 * (r & 1) + lane] = u;
    }
    for (int q = w; q < 4; q += nw) {  // both copies: cells outside the arrays are never polled
      const U2 u = load_u(q < 2 ? y0 - 2 + q : y0 + H + q - 2);
      for (int par = 0; par < 2; par++)
        reinterpret_cast<U2*>((q < 2 ? halo_b : halo_t) + par * PAIR)[32 * (q & 1) + lane] = u;
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
          e.y = (uint32_t)(own - urows) + chip_pair_off<T>(pq, npairs, 0) + ((r & 1) * 32 + col) * 2 * US;
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
          e.y = ((uint32_t)((below ? halo_b : halo_t) - urows) + (r * 32 + lane) * 2 * US) | 1;
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

    const char* rd_below = w > 0 ? own - ppw * PAIR + (npairs == 1 ? 0 : 2 * PAIR) : halo_b;
    const char* rd_above = w < nw - 1 ? own + ppw * PAIR : halo_t;
    const bool interior = x0 - 2 >= 1 && x0 + 29 <= nx - 3 && jA >= 3 && jA + rows <= ny - 2;
    const size_t rim_parity = (size_t)(ncx * ncy) * cells * RIM_BYTES;
    int it = 0;
    for (;; it++) {
      const int par = it & 1;
      if (jA < ny) {
        const char* below = rd_below + par * PAIR;
        const char* above = rd_above + par * PAIR;
        auto march = [&](auto plastic_c) {
          constexpr bool P = decltype(plastic_c)::value;
          auto rows_of = [&](auto np_c) {
            constexpr int NP = decltype(np_c)::value;
            auto run = [&](auto edge_c) {
              constexpr bool EDGE = decltype(edge_c)::value;
              ChipIo<T, TV, EDGE, NP, FLY == 2 || sizeof(T) == 4> io;
              io.mats = mats;
              io.idx = idx + w * rows * 32 + lane;
              io.below = below;
              io.above = above;
              io.own = own;
              io.rd = below;
              io.npairs = NP ? NP : npairs;
              io.par = par;
              io.right = lane < 31 ? 1 : 0;
              io.rows_left = ny - jA;
              io.col_own = col_own;
              io.vmem = vmem;
              io.yielded = yielded + lane;
              pair_march<T, TV, P, EDGE, NP, TRACK, kChipUnroll>(g, io, npairs, i, jA);
            };
            if (interior) run(std::false_type{});
            else run(std::true_type{});
          };
          if (npairs == 1) rows_of(std::integral_constant<int, 1>{});
          else if (npairs == 2) rows_of(std::integral_constant<int, 2>{});
          else if (npairs == 3) rows_of(std::integral_constant<int, 3>{});
          else rows_of(std::integral_constant<int, 0>{});
          tmem_st_wait();
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
        RimRecord<T>::put(out + cell * RIM_BYTES,
                reinterpret_cast<const U2*>(own + chip_pair_off<T>(r >> 1, npairs, par ^ 1))[(r & 1) * 32 + col], tag);
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
      for (int t0 = 0; t0 < npoll && !failed; t0 += FLY) {
        uint2 e[FLY];
        RimRecord<T> rec[FLY];
        bool wait[FLY];
#pragma unroll
        for (int k = 0; k < FLY; k++) {
          e[k].x = 0xffffffffu;
          if (t0 + k < npoll) e[k] = polls[(w * npoll + t0 + k) * 32 + lane];
          wait[k] = e[k].x != 0xffffffffu;
        }
        unsigned tries = 0;
        ChipClock clock;
        for (;;) {
          bool any = false;
#pragma unroll
          for (int k = 0; k < FLY; k++)
            if (wait[k]) rec[k].get(in + (size_t)e[k].x * RIM_BYTES);
#pragma unroll
          for (int k = 0; k < FLY; k++) {
            if (wait[k]) wait[k] = !rec[k].ready(tag);
            any |= wait[k];
          }
          if (!__any_sync(0xffffffffu, any)) break;
          if ((++tries & 1023u) == 0) {  // bounded: look at the clock and the state word now and then
            if (chip_look(job, clock.look(), a.start_ns, a.records_ns)) {
              failed = 1;
              break;
            }
          }
        }
#pragma unroll
        for (int k = 0; k < FLY; k++) {
          if (e[k].x == 0xffffffffu) continue;
          const uint32_t off = (e[k].y & ~1u) + ((e[k].y & 1u) ? (uint32_t)(par ^ 1) * PAIR : 0u);
          *reinterpret_cast<U2*>(urows + off) = rec[k].value();
        }
      }
      if (group_barrier_or(1 + group, 32 * nw, failed)) {
        // (which way out decides how the march comes out at 128 registers: 1024^2 9.98 us with break, 10.05 with
        // goto, a mixed batch 254 / 259 ms; tracking 1024^2 10.8 / 10.45)
        if (TRACK) goto leave;
        break;
      }
    }

    // back to global memory, unless the launch has failed: U of the last copy written, V
    if ((TRACK || it + 1 >= n_iter) && jA < ny) {
      __syncwarp();
      T* uxo = u_field<T>(f, false, src ^ (n_iter & 1));
      T* uyo = u_field<T>(f, true, src ^ (n_iter & 1));
      const int par = (it & 1) ^ 1;
      for (int q = 0; q < npairs; q++) {
        VPair<TV> v;
        tmem_ld(vmem + q * VW, v.w);
        tmem_ld_wait(v.w);
        for (int r = 0; r < 2; r++) {
          const int j = jA + 2 * q + r;
          if (col_own && j < ny) {
            const U2 u = reinterpret_cast<const U2*>(own + chip_pair_off<T>(q, npairs, par))[32 * r + lane];
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
leave:
  __syncthreads();
  if (wc == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(s_tmem));
}

// the kernels (ep2d_chip_kernels.cu) for a shape's warps per CTA and rows per warp
const void* chip_kernel_fp64(bool plastic, int warps, int rows);
const void* chip_kernel_mixed(bool plastic, int warps, int rows);
const void* chip_kernel_track(bool mixed, int warps, int rows);  // plastic
const void* chip_kernel_f32(bool plastic);
const void* chip_kernel_jobs(bool mixed);  // several RVEs

}  // namespace ep2d
