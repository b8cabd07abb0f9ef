// Truncated-spectra passes (spectral.cuh) and the filter operator for Fourier
// axes of any 2^a 3^b 5^c length up to 4096 (mr_spec.cu).  Same wide-row
// layout and pass contracts as the power-of-two kernels, so a grid may mix
// both kinds of axes, each on its own kernels.
//
// Pencils sit in shared memory and are transformed in place: forward
// decimation in frequency, inverse decimation in time, with radices up to 16
// held in registers (2160 = 16 15 9 and 3840 = 16 16 15 take three passes,
// one barrier each, where the radix-4/3/5/2 Stockham passes of
// mixed_radix.cu take seven and six with two).  Nothing is reordered: the
// spectrum is digit-reversed in place, and a pass finds the place of a point
// or mode from its digits (a few multiplications by float reciprocals; tables
// of places missed the small L1 left beside the shared memory).
//
// Measured per RK4 step against the Stockham passes: 3840 x 2160 12.2 -> 3.56
// ms (x pass 390, last pass 300, the two filter passes 732 us; the transforms
// are bound by instruction issue and shared-memory latency at 12-16 warps per
// SM, HBM at 15%), mixed 2D and 3D grids of 10^4 to 10^6 points 2.0 to 4.6
// times faster.
#pragma once
#include "spectral.cuh"

namespace ps {

struct SpecAxis {
  int n, km, nst;
  int radix[8];               // of pass s
  int m[8];                   // product of the later radices
  float inv_m[8], inv_r[8];   // 1 / m, 1 / radix
  const float2* tw;           // twiddles of the passes, spec_twiddles
  int len;                    // shared-memory elements of a pencil
  int st[8];                  // element stride of pass s's digit
  const float* P;
  const float* d;
};

// Radices (descending) of the fewest passes; false if n is not 5-smooth.
bool spec_factor(int n, int* radix, int* nst);
// Shared-memory layout of a pencil: point i = sum of digits q_s times the
// lengths below them sits at sum q_s st[s].  The strides are odd above the
// last digit, so a pass's accesses (linear in its own digit) and those of the
// last pass, whose threads differ in the higher digits, spread over the banks.
void spec_layout(const int* radix, int nst, int* len, int* st);

// Twiddles, pass after pass: W_L^{i q} at n - L + (q - 1) m + i for the pass of
// block length L = R m (n - 1 entries in all).  Consecutive butterflies read
// consecutive entries; taken from one table W_n^k at i q n / L they fell on
// one shared-memory bank from the second pass on.
void spec_twiddles(int n, const int* radix, int nst, float2* tw);

struct MrFilterArgs {
  const float* in;
  float* out;         // may alias in
  int nf;
  long fs, ss_in, ss_out;
  long es, npen;      // element stride along the pencil, pencils per field
  const int* active;
  const float* eadd;  // nullable: per-solve value added to the last field
};

cudaError_t launch_mrs_x(int nd, bool inc, bool flux, const SpecXArgs& a, const SpecAxis& ax, cudaStream_t s);
cudaError_t launch_mrs_f(const SpecFArgs& a, const SpecAxis& ax, cudaStream_t s);
cudaError_t launch_mrs_c(const SpecCArgs& a, const SpecAxis& ax, cudaStream_t s);
cudaError_t launch_mrs_i(const SpecIArgs& a, const SpecAxis& ax, cudaStream_t s);
// out = in - IFFT((1/n - P) FFT in) on nf fields (the end-of-step filter)
cudaError_t launch_mrs_filter(const MrFilterArgs& a, const SpecAxis& ax, int nsolve, cudaStream_t s);
// whether the x pass of nc components fits a CTA's shared memory
bool mrs_x_fits(int nd, int n);

}  // namespace ps
