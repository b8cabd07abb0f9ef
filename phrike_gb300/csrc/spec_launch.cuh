// Launchers of the truncated-spectra passes (spectral.cuh), instantiated per
// pencil length in kern_spec_n*.cu.
#pragma once
#include "launch.cuh"
#include "spectral.cuh"

namespace ps {

// Columns per CTA of the strided passes: the largest of 16, 8 and 4 (8 and 4
// at 1024 points; a CTA has at least one full warp) that gives two CTAs per
// SM.  A pencil's arithmetic does not depend on it.
template <int NN, typename F>
cudaError_t dispatch_spec_cols(int ncol, long outer, F&& f) {
  constexpr int TMAX = (NN >= 1024) ? 8 : 16;
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
  k_spec_x<NN, T, ND, PHYS, INC, FLUX><<<(a.nrow + T - 1) / T, Shape<NN>::A * T, sm, s>>>(a);
  return cudaGetLastError();
}
template <int NN, int T, int ND, int PHYS>
cudaError_t spec_x_mode(bool inc, bool flux, const SpecXArgs& a, cudaStream_t s) {
  if (inc && flux) return spec_x_T<NN, T, ND, PHYS, true, true>(a, s);
  if (inc) return spec_x_T<NN, T, ND, PHYS, true, false>(a, s);
  return spec_x_T<NN, T, ND, PHYS, false, true>(a, s);
}

#define PS_DEFINE_SPEC_LAUNCHERS(NN)                                                                  \
  template <>                                                                                         \
  cudaError_t launch_spec_f<NN>(const SpecFArgs& a, int planes, cudaStream_t s) {                     \
    return dispatch_spec_cols<NN>(a.ncol, planes, [&](auto tw) -> cudaError_t {                       \
      constexpr int T = decltype(tw)::value;                                                          \
      const size_t sm = sizeof(SpecSmem<NN, T>);                                                      \
      cudaError_t e;                                                                                  \
      if ((e = set_smem(k_spec_f<NN, T>, sm)) != cudaSuccess) return e;                               \
      k_spec_f<NN, T><<<dim3((a.ncol + T - 1) / T, planes), Shape<NN>::A * T, sm, s>>>(a);            \
      return cudaGetLastError();                                                                      \
    });                                                                                               \
  }                                                                                                   \
  template <>                                                                                         \
  cudaError_t launch_spec_c<NN>(const SpecCArgs& a, int nsol, cudaStream_t s) {                       \
    return dispatch_spec_cols<NN>(a.ncol, (long)nsol * a.nouter, [&](auto tw) -> cudaError_t {        \
      constexpr int T = decltype(tw)::value;                                                          \
      const size_t sm = sizeof(SpecSmem<NN, T>);                                                      \
      cudaError_t e;                                                                                  \
      if ((e = set_smem(k_spec_c<NN, T>, sm)) != cudaSuccess) return e;                               \
      k_spec_c<NN, T><<<dim3((a.ncol + T - 1) / T, nsol * a.nouter), Shape<NN>::A * T, sm, s>>>(a);   \
      return cudaGetLastError();                                                                      \
    });                                                                                               \
  }                                                                                                   \
  template <>                                                                                         \
  cudaError_t launch_spec_i<NN>(const SpecIArgs& a, int planes, cudaStream_t s) {                     \
    return dispatch_spec_cols<NN>(a.ncol, planes, [&](auto tw) -> cudaError_t {                       \
      constexpr int T = decltype(tw)::value;                                                          \
      const size_t sm = sizeof(SpecSmem<NN, T>);                                                      \
      cudaError_t e;                                                                                  \
      if ((e = set_smem(k_spec_i<NN, T>, sm)) != cudaSuccess) return e;                               \
      k_spec_i<NN, T><<<dim3((a.ncol + T - 1) / T, planes), Shape<NN>::A * T, sm, s>>>(a);            \
      return cudaGetLastError();                                                                      \
    });                                                                                               \
  }

// Euler x pass of every length, MHD x pass in a unit of its own
#define PS_DEFINE_SPEC_X(NN, PHYS)                                                                    \
  template <>                                                                                         \
  cudaError_t launch_spec_x<NN, PHYS>(int nd, bool inc, bool flux, const SpecXArgs& a, cudaStream_t s) { \
    return dispatch_rows<NN>(a.nrow, [&](auto tw) -> cudaError_t {                                    \
      constexpr int T = decltype(tw)::value;                                                          \
      if (nd == 3) {                                                                                  \
        if constexpr (PHYS == 1 && NN > 256) return cudaErrorInvalidValue; /* 3D MHD: 8..256 */       \
        else return spec_x_mode<NN, T, 3, PHYS>(inc, flux, a, s);                                     \
      }                                                                                               \
      return spec_x_mode<NN, T, 2, PHYS>(inc, flux, a, s);                                            \
    });                                                                                               \
  }

}  // namespace ps
