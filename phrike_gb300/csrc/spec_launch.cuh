// Launchers of the truncated-spectra passes (spectral.cuh), instantiated per
// pencil length in kern_spec_n*.cu.
#pragma once
#include <atomic>

#include "launch.cuh"
#include "spectral.cuh"

namespace ps {

// Columns per CTA of the strided passes: the largest of 16, 8 and 4 (8 and 4
// at 1024 points; a CTA has at least one full warp) that gives two CTAs per
// SM.  A pencil's arithmetic does not depend on it.
template <int NN, typename F>
cudaError_t dispatch_spec_cols(int ncol, long outer, F&& f) {
  constexpr int TMAX = (NN >= 512) ? 8 : 16;
  constexpr int TMIN = cmax_int(4, 32 / Shape<NN>::A);
  if constexpr (TMAX >= 16 && TMIN < 16)
    if ((ncol + 15) / 16 * outer >= 2L * 148) return f(std::integral_constant<int, 16>{});
  if constexpr (TMIN < 8 && TMAX >= 8)
    if ((ncol + 7) / 8 * outer >= 2L * 148) return f(std::integral_constant<int, 8>{});
  return f(std::integral_constant<int, TMIN>{});
}

template <int NN, int T, int ND, int PHYS, bool INC, bool FLUX>
cudaError_t spec_x_T(const SpecXArgs& a, cudaStream_t s) {
  const size_t sm = sizeof(SpecXSmem<NN, T>);
  cudaError_t e;
  if ((e = set_smem(k_spec_x<NN, T, ND, PHYS, INC, FLUX>, sm)) != cudaSuccess) return e;
  return launch_dep(k_spec_x<NN, T, ND, PHYS, INC, FLUX>, (a.rows + T - 1) / T, Shape<NN>::A * T, sm, s, a);
}
template <int NN, int T, int ND, int PHYS>
cudaError_t spec_x_mode(bool inc, bool flux, const SpecXArgs& a, cudaStream_t s) {
  if (inc && flux) return spec_x_T<NN, T, ND, PHYS, true, true>(a, s);
  if (inc) return spec_x_T<NN, T, ND, PHYS, true, false>(a, s);
  return spec_x_T<NN, T, ND, PHYS, false, true>(a, s);
}

// A walking grid: as many CTAs as fit the GPU at once, or one per tile.
template <int NN, int T, typename K>
cudaError_t spec_grid(K kernel, int threads, size_t sm, long items, int* grid) {
  static std::atomic<int> known{0};  // per kernel and shape (one instantiation of this function each)
  int resident = known.load();
  if (resident == 0) {
    int per = 0, dev = 0, sms = 0;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, threads, sm);
    if (e == cudaSuccess) e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    if (per < 1) return cudaErrorInvalidConfiguration;
    known.store(resident = per * sms);
  }
  *grid = (int)(items < resident ? items : resident);
  return cudaSuccess;
}

#define PS_DEFINE_SPEC_STRIDED(NN, NAME, ARGS, KERNEL, SMEM, OUTER)                                   \
  template <>                                                                                         \
  cudaError_t NAME<NN>(const ARGS& a, cudaStream_t s) {                                               \
    return dispatch_spec_cols<NN>(a.ncol, OUTER, [&](auto tw) -> cudaError_t {                        \
      constexpr int T = decltype(tw)::value;                                                          \
      const size_t sm = sizeof(SMEM<NN, T>);                                                                \
      cudaError_t e;                                                                                  \
      int grid;                                                                                       \
      if ((e = set_smem(KERNEL<NN, T>, sm)) != cudaSuccess) return e;                                 \
      auto* k = KERNEL<NN, T>;                                                                        \
      const long items = (long)((a.ncol + T - 1) / T) * (OUTER);                                      \
      if ((e = spec_grid<NN, T>(k, Shape<NN>::A * T, sm, items, &grid)) != cudaSuccess) return e;     \
      return launch_dep(k, grid, Shape<NN>::A * T, sm, s, a);                                         \
    });                                                                                               \
  }
#define PS_DEFINE_SPEC_LAUNCHERS(NN)                                                                  \
  PS_DEFINE_SPEC_STRIDED(NN, launch_spec_f, SpecFArgs, k_spec_f, SpecPairSmem, (long)a.planes) \
  PS_DEFINE_SPEC_STRIDED(NN, launch_spec_c, SpecCArgs, k_spec_c, SpecPairSmem, (long)a.nouter * a.nsolve) \
  PS_DEFINE_SPEC_STRIDED(NN, launch_spec_i, SpecIArgs, k_spec_i, SpecISmem, (long)a.planes)

// Euler x pass of every length, MHD x pass in a unit of its own
#define PS_DEFINE_SPEC_X(NN, PHYS)                                                                    \
  template <>                                                                                         \
  cudaError_t launch_spec_x<NN, PHYS>(int nd, bool inc, bool flux, const SpecXArgs& a, cudaStream_t s) { \
    return dispatch_rows<NN>(a.rows, [&](auto tw) -> cudaError_t {                                    \
      constexpr int T = decltype(tw)::value;                                                          \
      if (nd == 3) {                                                                                  \
        if constexpr (PHYS == 1 && NN > 256) return cudaErrorInvalidValue; /* 3D MHD: 8..256 */       \
        else return spec_x_mode<NN, T, 3, PHYS>(inc, flux, a, s);                                     \
      }                                                                                               \
      return spec_x_mode<NN, T, 2, PHYS>(inc, flux, a, s);                                            \
    });                                                                                               \
  }

}  // namespace ps
