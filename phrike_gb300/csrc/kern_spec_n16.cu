// Truncated-spectra passes for pencils of 16 points: strided passes and the
// Euler x pass (the MHD x pass is in kern_specm_n16.cu).
#include "spec_launch.cuh"

namespace ps {
PS_DEFINE_SPEC_LAUNCHERS(16)
PS_DEFINE_SPEC_X(16, 0)
}  // namespace ps
