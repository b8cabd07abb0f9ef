// Truncated-spectra passes for pencils of 256 points: strided passes and the
// Euler x pass (the MHD x pass is in kern_specm_n256.cu).
#include "spec_launch.cuh"

namespace ps {
PS_DEFINE_SPEC_LAUNCHERS(256)
PS_DEFINE_SPEC_X(256, 0)
}  // namespace ps
