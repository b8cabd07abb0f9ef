// Launchers of the truncated-spectra passes (spectral.cuh), instantiated per
// pencil length in kern_spec_n*.cu.
#pragma once
#include <atomic>

#include "launch.cuh"
#include "spectral.cuh"

namespace ps {

// Columns per CTA of the strided passes: asked for (ps_plan_desc.tile_cols, the
// nearest width that is built), or the largest of 16, 8 and 4 (8 and 4 from 512
// points; a CTA has at least one full warp) that gives two CTAs per SM.  A
// pencil's arithmetic does not depend on it.
template <int NN, typename F>
cudaError_t dispatch_spec_cols(int ncol, long outer, int asked, F&& f) {
  constexpr int TMAX = (NN >= 512) ? 8 : 16;
  constexpr int TMIN = cmax_int(4, 32 / Shape<NN>::A);
  auto take = [&](int T) { return asked > 0 ? asked >= T : (ncol + T - 1) / T * outer >= 2L * 148; };
  if constexpr (TMAX >= 16 && TMIN < 16)
    if (take(16)) return f(std::integral_constant<int, 16>{});
  if constexpr (TMIN < 8 && TMAX >= 8)
    if (take(8)) return f(std::integral_constant<int, 8>{});
  return f(std::integral_constant<int, TMIN>{});
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

template <int NN, int ND, int PHYS, bool INC, bool FLUX>
cudaError_t spec_xs(const SpecXArgs& a, cudaStream_t s) {
  constexpr int T = 32 / Shape<NN>::A, NG = (ND == 3 && PHYS == 0) ? 3 : 4, NC = (PHYS == 1) ? 8 : ND + 2;
  const size_t sm = sizeof(SpecXsSmem<NN, T, NC, NG>);
  auto* k = k_spec_xs<NN, ND, PHYS, NG, INC, FLUX>;
  cudaError_t e;
  int grid = (a.rows + T - 1) / T;
  if ((e = set_smem(k, sm)) != cudaSuccess) return e;
  if (PHYS == 1 &&  // these kernels walk over their tiles
      (e = spec_grid<NN, (PHYS * 4 + ND) * 4 + INC * 2 + FLUX>(k, 32 * NG, sm, grid, &grid)) != cudaSuccess)
    return e;
  return launch_dep(k, grid, 32 * NG, sm, s, a);
}
template <int NN, int ND, int PHYS>
cudaError_t spec_xs_mode(bool inc, bool flux, const SpecXArgs& a, cudaStream_t s) {
  if (inc && flux) return spec_xs<NN, ND, PHYS, true, true>(a, s);
  if (inc) return spec_xs<NN, ND, PHYS, true, false>(a, s);
  return spec_xs<NN, ND, PHYS, false, true>(a, s);
}

#define PS_DEFINE_SPEC_STRIDED(NN, NAME, ARGS, KERNEL, SMEM, OUTER)                                   \
  template <>                                                                                         \
  cudaError_t NAME<NN>(const ARGS& a, cudaStream_t s) {                                               \
    return dispatch_spec_cols<NN>(a.ncol, OUTER, a.tile, [&](auto tw) -> cudaError_t {                \
      constexpr int T = decltype(tw)::value;                                                          \
      const size_t sm = sizeof(SMEM<NN, T>);                                                          \
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

// Euler rows of k_spec_x fill 32 / A pencils per warp; up to eight such warps
// per SM their chains of 6 to 12 transforms do not overlap enough, and the jobs
// of a row go to several warps (k_spec_xs).  Step times, k_spec_x against
// k_spec_xs: KHI 128^2 84.1 -> 65.7 us (32 warps), Taylor-Green 64^3 94.9 ->
// 92.8 us (1024), batches at 6.7 warps per SM between 52 -> 46 us (64^2 x 64)
// and 90 -> 92 us (256^2 x 8); at 10 to 27 warps per SM k_spec_xs takes 1% to
// 13% longer (256^2 x 32 237 against 267 us) but at 512^2 x 4 (208 against
// 199 us).  MHD rows up to 512 points always take k_spec_xs: Orszag-Tang 512^2
// 249 -> 183 us (512 warps), 3D MHD 128^3 1184 -> 1056 us (4096).  A batch may
// take the other kernel than one of its solves alone: both give the same bits.
constexpr long kSpecXsWarps = 8 * 152;

// Euler x pass of every length, MHD x pass in a unit of its own
#define PS_DEFINE_SPEC_X(NN, PHYS)                                                                    \
  template <>                                                                                         \
  cudaError_t launch_spec_x<NN, PHYS>(int nd, bool inc, bool flux, const SpecXArgs& a, cudaStream_t s) { \
    constexpr bool few = Shape<NN>::A <= 32; /* a warp holds a pencil */                              \
    if constexpr (few && PHYS == 1) {                                                                 \
      if (nd == 2) return spec_xs_mode<NN, 2, 1>(inc, flux, a, s);                                    \
      if constexpr (NN <= 256) return spec_xs_mode<NN, 3, 1>(inc, flux, a, s); /* 3D MHD: 8..256 */   \
      return cudaErrorInvalidValue;                                                                   \
    } else {                                                                                          \
      if constexpr (few)                                                                              \
        if ((long)a.rows * Shape<NN>::A <= 32 * kSpecXsWarps)                                         \
          return nd == 2 ? spec_xs_mode<NN, 2, 0>(inc, flux, a, s) : spec_xs_mode<NN, 3, 0>(inc, flux, a, s); \
      return dispatch_rows<NN>(a.rows, [&](auto tw) -> cudaError_t {                                  \
        constexpr int T = decltype(tw)::value;                                                        \
        if (nd == 2) return spec_x_mode<NN, T, 2, PHYS>(inc, flux, a, s);                             \
        if constexpr (PHYS == 0) return spec_x_mode<NN, T, 3, PHYS>(inc, flux, a, s);                 \
        else return cudaErrorInvalidValue;                                                            \
      });                                                                                             \
    }                                                                                                 \
  }

}  // namespace ps
