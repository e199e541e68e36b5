// ep2d_chip.cu -- launches of the on-chip form (ep2d_iter_chip.cuh; its kernels: ep2d_chip_kernels.cu).
#include <algorithm>

#include "ep2d_iter_chip.cuh"

namespace ep2d {

// The shape of the on-chip form for a grid.  Rows first: the fewest rows per warp (a march
// of R rows costs R + 3 row steps, and a warp's latency sets the time of a small grid) for
// which every tile finds a place among CHIP_SMS CTAs of CHIP_WARPS warps.  Then the fewest
// warps per SM, in tiles of at least 4 warps, and more tiles per CTA rather than fewer: while one
// waits for its neighbours' rims another computes (1024^2, us an iteration: 4 tiles of
// 4 warps 9.9, 2 of 8 10.3, 1 of 16 10.7; 512^2, 6 rows: 3 of 4 4.27, 2 of 6 4.34, 4 of 4 4.78;
// 256^2, 2 rows: 2 of 5 2.70, 2 of 7 2.89, 1 of 10 2.85).
ChipShape chip_shape(int nx, int ny) {
  ChipShape best;
  const int ncx = (nx + STREAM_COLS - 1) / STREAM_COLS;
  for (int rows = 2; rows <= 18 && !best.warps; rows += 2) {
    int best_cost = 1 << 30;
    for (int groups = 1; groups <= 4; groups++)
      for (int warps = 4; groups * warps <= CHIP_WARPS; warps++) {
        const int ncy = (ny + warps * rows - 1) / (warps * rows);
        if ((int64_t)ncx * ncy > (int64_t)CHIP_SMS * groups || chip_smem_bytes(groups, warps, rows) > CHIP_SMEM)
          continue;
        const int cost = groups * warps + (groups == 1 ? 1 : 0);  // warps per SM
        if (cost <= best_cost) {
          best_cost = cost;
          best.warps = warps;
          best.rows = rows;
          best.groups = groups;
          best.ncx = ncx;
          best.ncy = ncy;
        }
      }
  }
  return best;
}

// Beside other grids: the shape with which the most iterations per second are run if the others are like
// this one.  An iteration takes 1.75 + 0.0325 us per row and warp of a CTA (measured, FP64 with the return map:
// 2 rows x 4 warps 2.05, 2 x 10 2.54, 6 x 12 3.8, 10 x 16 6.8, 16 x 16 10.0), of which the first part overlaps.
ChipShape chip_shape_beside(int nx, int ny, int rves, int sms) {
  auto at_once = [&](const ChipShape& s) {
    return std::min(rves, sms / chip_ctas(nx, ny, s.groups, s.warps, s.rows));
  };
  auto rate = [&](const ChipShape& s) { return at_once(s) / (1.75 + 0.0325 * s.rows * s.groups * s.warps); };
  // the shape it takes alone where none lets more of them run at once (two handles: 768^2 6.9 us, 7.3 in
  // shapes the line above likes better; 1024^2 10.0, 10.9)
  ChipShape best, s = chip_shape(nx, ny);
  const int alone = s.warps ? at_once(s) : 0;
  double most = alone ? rate(s) : 0.0;
  if (alone) best = s;
  for (s.rows = 2; s.rows <= 18; s.rows += 2)
    for (s.groups = 1; s.groups <= 4; s.groups++)
      for (s.warps = 4; s.groups * s.warps <= CHIP_WARPS; s.warps++) {
        if (chip_smem_bytes(s.groups, s.warps, s.rows) > CHIP_SMEM || at_once(s) <= alone || rate(s) <= most) continue;
        most = rate(s);
        best = s;
      }
  return best;
}

size_t chip_rim_bytes(int nx, int ny, int warps, int rows, bool f32) {
  const size_t ncx = (nx + STREAM_COLS - 1) / STREAM_COLS, ncy = (ny + warps * rows - 1) / (warps * rows);
  return 2 * (f32 ? RimRecord<float>::BYTES : RimRecord<double>::BYTES) * ncx * ncy * (4 * (size_t)warps * rows + 4 * STREAM_COLS);
}

// 4 records per row of padded height and 4 x STREAM_COLS per tile: the shortest tiles of at
// least 4 warps, and the tallest padding, decide
size_t chip_rim_capacity(int nx, int ny) {
  const ChipShape s = chip_shape(nx, ny);
  size_t most = 0;
  if (s.warps)
    for (int rows = s.rows; rows <= 18; rows += 2)
      for (int warps = 4; warps <= CHIP_WARPS; warps++) most = std::max(most, chip_rim_bytes(nx, ny, warps, rows));
  return most;
}

int chip_ctas(int nx, int ny, int groups, int warps, int rows) {
  const int ncx = (nx + STREAM_COLS - 1) / STREAM_COLS, ncy = (ny + warps * rows - 1) / (warps * rows);
  return (ncx * ncy + groups - 1) / groups;
}
size_t chip_smem(int groups, int warps, int rows, bool track) { return chip_smem_bytes(groups, warps, rows, track); }

namespace {
// the FP64 (mixed: FP32 velocities) kernel of one RVE for a shape of `warps` warps per CTA
const void* chip_kernel(bool plastic, bool mixed, bool track, int warps, int rows) {
  if (track) return chip_kernel_track(mixed, warps, rows);
  return mixed ? chip_kernel_mixed(plastic, warps, rows) : chip_kernel_fp64(plastic, warps, rows);
}

template <int JOBS>
cudaError_t launch_chip_jobs(const ChipJob* jobs, int njobs, const void* kern, const ChipShape& s, int n_iter, int blocks,
                             const ChipWaits& waits, cudaStream_t stream, bool track = false) {
  ChipArgs<JOBS> a;
  a.njobs = njobs;
  a.warps = s.warps;
  a.rows = s.rows;
  a.n_iter = n_iter;
  a.start_ns = waits.start_ns;
  a.records_ns = waits.records_ns;
  std::copy(jobs, jobs + njobs, a.job);
  void* args[] = {&a};
  // (here rather than for every kernel when a device is first used: it loads the kernel's module)
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, CHIP_SMEM);
  if (e != cudaSuccess) return e;
  const size_t sm = std::max(chip_smem_bytes(s.groups, s.warps, s.rows, track), (size_t)CHIP_SMEM_MIN);
  return cudaLaunchCooperativeKernel(kern, dim3(blocks), dim3(32 * s.warps * s.groups), args, sm, stream);
}
}  // namespace

cudaError_t launch_iter_chip(ChipJob* jobs, int njobs, bool mixed, const ChipShape& s, int n_iter,
                             const ChipWaits& waits, cudaStream_t stream, bool track, bool f32) {
  if (njobs < 1 || njobs > CHIP_JOBS || ((track || f32) && njobs > 1) || n_iter < 2 || s.warps < 1 || s.groups < 1 ||
      s.warps * s.groups > CHIP_WARPS || s.rows < 2 || s.rows > 18 || (s.rows & 1) ||
      chip_smem_bytes(s.groups, s.warps, s.rows, track) > CHIP_SMEM)
    return cudaErrorInvalidValue;
  int blocks = 0;
  for (int k = 0; k < njobs; k++) {
    ChipJob& j = jobs[k];
    if (!j.rim || !j.state) return cudaErrorInvalidValue;
    j.ncx = (j.g.nx + STREAM_COLS - 1) / STREAM_COLS;
    j.ncy = (j.g.ny + s.warps * s.rows - 1) / (s.warps * s.rows);
    j.cta0 = blocks;
    const cudaError_t e = cudaMemsetAsync(j.rim, 0, chip_rim_bytes(j.g.nx, j.g.ny, s.warps, s.rows, f32), stream);
    if (e != cudaSuccess) return e;
    const int ctas = (j.ncx * j.ncy + s.groups - 1) / s.groups;
    blocks += ctas;
    j.full = j.count0 + ctas;
  }
  const int missing = std::min(waits.missing, blocks - jobs[njobs - 1].cta0 - 1);  // of the last job
  blocks -= missing;
  if (waits.missing_started) jobs[njobs - 1].full -= missing;
  if (njobs == 1) {
    const bool pl = jobs[0].plastic != 0;
    const void* kern = f32 ? chip_kernel_f32(pl) : chip_kernel(pl, mixed, track && pl, s.warps * s.groups, s.rows);
    return launch_chip_jobs<1>(jobs, 1, kern, s, n_iter, blocks, waits, stream, track && pl && !f32);
  }
  return launch_chip_jobs<CHIP_JOBS>(jobs, njobs, chip_kernel_jobs(mixed), s, n_iter, blocks, waits, stream);
}

}  // namespace ep2d
