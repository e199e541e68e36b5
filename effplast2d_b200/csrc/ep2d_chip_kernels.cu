// ep2d_chip_kernels.cu -- the instantiations of the on-chip form's kernel (ep2d_iter_chip.cuh), compiled once
// for each EP2D_CHIP_PART into a module of its own (without it, all into one).  A process loads a module
// when it first launches a kernel of it: with all of them in one file and their attributes set for the first
// handle, that handle and its first solve took 51 ms, with the parts 24 (64^2, NL=3, B200).
#include "ep2d_iter_chip.cuh"

namespace ep2d {

namespace {
template <int PLASTIC, typename TV, bool TRACK>
const void* chip_kernel_of(int warps, int rows) {
  if (warps <= 8) return (const void*)k_iter_chip<PLASTIC, 1, double, TV, TRACK, 8, 2>;
  if (warps <= 12) return (const void*)k_iter_chip<PLASTIC, 1, double, TV, TRACK, 12, 2>;
  if constexpr (PLASTIC == 1)
    if (rows >= 10) return (const void*)k_iter_chip<PLASTIC, 1, double, TV, TRACK, 16, 3>;
  return (const void*)k_iter_chip<PLASTIC, 1, double, TV, TRACK, 16, 2>;
}
}  // namespace

#if !defined(EP2D_CHIP_PART) || EP2D_CHIP_PART == 0
const void* chip_kernel_fp64(bool plastic, int warps, int rows) {
  return plastic ? chip_kernel_of<1, double, false>(warps, rows) : chip_kernel_of<0, double, false>(warps, rows);
}
#endif
#if !defined(EP2D_CHIP_PART) || EP2D_CHIP_PART == 1
const void* chip_kernel_mixed(bool plastic, int warps, int rows) {
  return plastic ? chip_kernel_of<1, float, false>(warps, rows) : chip_kernel_of<0, float, false>(warps, rows);
}
#endif
#if !defined(EP2D_CHIP_PART) || EP2D_CHIP_PART == 2
const void* chip_kernel_track(bool mixed, int warps, int rows) {
  return mixed ? chip_kernel_of<1, float, true>(warps, rows) : chip_kernel_of<1, double, true>(warps, rows);
}
#endif
#if !defined(EP2D_CHIP_PART) || EP2D_CHIP_PART == 3
const void* chip_kernel_f32(bool plastic) {
  return plastic ? (const void*)k_iter_chip<1, 1, float, float> : (const void*)k_iter_chip<0, 1, float, float>;
}
#endif
#if !defined(EP2D_CHIP_PART) || EP2D_CHIP_PART == 4
const void* chip_kernel_jobs(bool mixed) {
  return mixed ? (const void*)k_iter_chip<2, CHIP_JOBS, double, float> : (const void*)k_iter_chip<2, CHIP_JOBS, double, double>;
}
#endif

}  // namespace ep2d
